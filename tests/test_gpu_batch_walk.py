"""A batch on the near-first trees with a context that does not gain from them
renders what each context renders by itself."""
import numpy as np
import pytest

from zig_ornament_gb300 import ornament, scenes

pytestmark = pytest.mark.gpu


def _renderer(scene, builder, width, height, passes):
    r = ornament.Renderer(ornament.Bvh(scene, builder=builder), device=0)
    state = ornament.State()
    state.setDepth(8)
    state.setIterations(passes)
    r.set_state(state.to_struct())
    r.set_resolution(width, height)
    r.set_camera(scene.camera.to_struct())
    return r


def test_a_context_on_a_good_tree_among_others():
    def make():
        good = scenes.instanced_meshes_scene(61, 35, seed=3, n_blas=2, n_instances=24, tri_range=(8_000, 12_000),
                                             texture_size=32)
        others = scenes.instanced_meshes_scene(131, 77, seed=1, n_blas=3, n_instances=60, tri_range=(2_000, 5_000),
                                               texture_size=32)
        return [_renderer(good, "sah", 61, 35, 2), _renderer(others, "reference", 131, 77, 4),
                _renderer(scenes.spheres_scene(64, 48), "reference", 64, 48, 3)]
    alone, together = make(), make()
    trees = [r.near_trees() for r in together]
    assert trees[0] == 1 and min(trees[1:]) >= 2   # (the first does not gain)
    for r in alone:
        r.render()
    with_batch = ornament.Batch(together)
    with_batch.render()
    with_batch.synchronize()
    for a, b in zip(alone, together):
        for x, y in zip(a.progress()[:2], b.progress()[:2]):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
        assert np.array_equal(a.framebuffer().view(np.uint32), b.framebuffer().view(np.uint32))
    with_batch.close()
    for r in alone + together:
        r.close()
