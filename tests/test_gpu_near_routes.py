"""Which trees a context walks (orn_near_trees), for the scenes of
test_gpu_near.py and at the conditions under which the near-first trees are
not built or not taken: without this, a comparison of the two walks could be
one walk with itself."""
import numpy as np
import pytest

import test_gpu_near as near
from zig_ornament_gb300 import ornament, scenes

pytestmark = pytest.mark.gpu


def _trees(bvh):
    r = ornament.Renderer(bvh, device=0)
    n = r.near_trees()
    r.close()
    return n


@pytest.mark.parametrize("name", near.SCENES)
def test_scenes_have_near_first_trees(name):
    assert _trees(ornament.Bvh(near.SCENES[name]())) > 0


@pytest.mark.parametrize("change", ["wide_leaf", "child_outside"])
def test_other_boxes_have_none(change):
    bvh = ornament.Bvh(near.SCENES["mixed"]())
    inner = np.nonzero(bvh.blas_nodes["node_type"] == 0)[0]
    if change == "wide_leaf":
        kinds = bvh.blas_nodes["node_type"][bvh.blas_nodes["left_or_custom_id"][inner]]
        bvh.blas_nodes["left_aabb_min_or_v0"][inner[kinds == 3][0]] -= 0.05
    else:
        bvh.blas_nodes["left_aabb_max_or_v1"][inner[-1]] -= 0.2
    assert _trees(bvh) == 0


@pytest.mark.parametrize("needles,some", [(64, True), (65, False)])
def test_many_slivers_have_none(needles, some):
    s = ornament.Scene()
    rs = np.random.default_rng(5)
    t = rs.uniform(-2, 2, (200, 1, 3)) + rs.uniform(0.2, 0.6, (200, 3, 3)) * np.eye(3)
    t[:needles, 2] = 0.5 * (t[:needles, 0] + t[:needles, 1]) + 1e-5
    near._mesh(s, t)
    assert (_trees(ornament.Bvh(s)) > 0) == some


@pytest.mark.parametrize("builder,trees", [("reference", 3), ("sah", 1), ("lbvh", 1)])
def test_large_scenes_by_their_trees(builder, trees):
    scene = scenes.instanced_meshes_scene(97, 53, seed=3, n_blas=2, n_instances=24, tri_range=(8_000, 12_000),
                                          texture_size=32)
    assert _trees(ornament.Bvh(scene, builder=builder)) == trees
