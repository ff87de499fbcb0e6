"""Several threads, a context each, make the first launches of a process at
once: every one gets what a single thread gets."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = r"""
import sys, threading
import numpy as np
from zig_ornament_gb300 import ornament, scenes

def work(r, scene):
    rays = np.concatenate([np.random.default_rng(1).uniform(-6, 6, (500, 3)),
                           np.random.default_rng(2).normal(size=(500, 3))], 1).astype(np.float32)
    hits, _ = r.trace_rays(rays, with_visits=False)
    r.set_camera(scene.camera.to_struct())
    r.render()
    return hits.tobytes() + r.framebuffer().tobytes()

def make():
    scene = scenes.small_test_scene(48, 32)
    r = ornament.Renderer(ornament.Bvh(scene), device=0)
    state = ornament.State()
    state.setIterations(2)
    r.set_state(state.to_struct())
    r.set_resolution(48, 32)
    return r, scene

made = [make() for _ in range(8)]
results, barrier = [None] * 8, threading.Barrier(8)
def run(i):
    barrier.wait()
    results[i] = work(*made[i])
threads = [threading.Thread(target=run, args=(i,)) for i in range(8)]
for t in threads: t.start()
for t in threads: t.join()
alone = work(*make())
sys.exit(0 if all(x == alone for x in results) else 1)
"""


@pytest.mark.parametrize("time", range(3))
def test_first_launches_of_several_threads(time):
    assert subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, timeout=120).returncode == 0
