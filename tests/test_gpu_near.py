"""The near-first trees (csrc/tree_build.cu, csrc/pt_near.cuh) give the
reference walk's results bit for bit: closest hits against the walk that
counts visits, pictures against counting renders (both keep the reference's
tree and order), at the forms where the two could part — ties, flat boxes,
slivers, one-primitive scenes, rays from far away and along axes — and blobs
that the trees are not built for."""
import numpy as np
import pytest

from zig_ornament_gb300 import _lib, ornament, scenes
from zig_ornament_gb300.ornament import F32, identity, mul, scaling, translation

pytestmark = pytest.mark.gpu


def _mesh(scene, triangles, transform=None, material=None):
    v = np.concatenate([np.asarray(triangles, F32).reshape(-1, 3), np.ones((3 * len(triangles), 1), F32)], 1)
    idx = np.arange(len(v), dtype=np.uint32)
    n = np.tile(np.array([0, 1, 0, 0], F32), (len(v), 1))
    return scene.createMesh(v, idx, n, idx, np.zeros((0, 2), F32), np.zeros(0, np.uint32),
                            identity() if transform is None else transform,
                            material or scene.lambertian((0.5, 0.5, 0.5, 1.0)))


def _one_triangle():
    s = ornament.Scene()
    _mesh(s, [[[0, 0, 0], [2, 0, 0], [0, 2, 0]]])
    return s


def _one_sphere():
    s = ornament.Scene()
    s.createSphere((0, 0, 0, 1), 1.5, s.lambertian((0.5, 0.5, 0.5, 1.0)))
    return s


def _copies():
    """The same triangles several times over, and coplanar overlapping ones: every hit is a tie."""
    s = ornament.Scene()
    t = [[[-2, -2, 0], [2, -2, 0], [0, 2, 0]]]
    m = _mesh(s, t * 5 + [[[-2, -2, 0], [2, -2, 0], [2, 2, 0]]])
    for k in range(3):
        s.createMeshInstance(m, identity(), s.materials[0])
    s.createMeshInstance(m, translation(0.5, 0.25, 0.0), s.materials[0])
    return s


def _slivers():
    """Needles (edges parallel to one part in 10^4) and zero-area triangles among ordinary ones."""
    s = ornament.Scene()
    rs = np.random.default_rng(3)
    t = rs.uniform(-2, 2, (60, 1, 3)) + rs.uniform(-0.6, 0.6, (60, 3, 3))
    t[:8, 2] = 0.5 * (t[:8, 0] + t[:8, 1]) + 1e-4 * rs.normal(size=(8, 3))
    t[8:10, 2] = t[8:10, 1]
    t[10:12, 1] = t[10:12, 0]
    m = _mesh(s, t)
    s.createMeshInstance(m, mul(scaling(0.3, 0.3, 0.3), translation(1, 1, 1)), s.materials[0])
    return s


def _needle_only():
    s = ornament.Scene()
    _mesh(s, [[[-2, 0, 0], [2, 0, 0], [0.1, 1e-4, 0]]])
    return s


def _scales():
    """Triangles over thirty powers of ten (a tree as deep as it has leaves)."""
    s = ornament.Scene()
    _mesh(s, [[[q, 0, 0], [1.2 * q, 0, 0.1 * q], [q, 0.3 * q, 0]] for q in 10.0 ** np.linspace(-3, 4, 40)])
    return s


SCENES = {"one_triangle": _one_triangle, "one_sphere": _one_sphere, "copies": _copies, "slivers": _slivers,
          "needle": _needle_only, "scales": _scales,
          "mixed": lambda: scenes.small_test_scene(96, 64), "spheres": scenes.spheres_scene,
          "room": scenes.cornell_box_scene,
          "instanced": lambda: scenes.instanced_meshes_scene(n_blas=4, n_instances=40, tri_range=(200, 3000),
                                                             texture_size=16)}


def _rays(extent, n=60_000, seed=5):
    rs = np.random.default_rng(seed)
    o, d = rs.uniform(-extent, extent, (n, 3)), rs.normal(size=(n, 3))
    k = n // 6
    d[:k, 1:] = 0.0                                   # along an axis
    d[k:2 * k] = -o[k:2 * k]                          # towards the middle, where copies and poles lie
    o[2 * k:2 * k + 50] *= 1e6                        # from far away
    d[2 * k:2 * k + 50] = -o[2 * k:2 * k + 50]
    o[3 * k:4 * k] = np.round(o[3 * k:4 * k])         # from lattice points
    d[3 * k:4 * k] = np.round(2 * d[3 * k:4 * k])
    d[(d == 0).all(1)] = (0, 0, 1)
    return np.concatenate([o, d], 1).astype(F32)


@pytest.mark.parametrize("triangle_test", [_lib.TRIANGLE_MOLLER_TRUMBORE, _lib.TRIANGLE_WATERTIGHT], ids=["mt", "wt"])
@pytest.mark.parametrize("name", SCENES)
def test_hits_equal_the_reference_walks(name, triangle_test):
    r = ornament.Renderer(ornament.Bvh(SCENES[name]()), device=0)
    state = ornament.State()
    state.triangle_test = triangle_test
    r.set_state(state.to_struct())
    rays = _rays({"instanced": 60.0, "spheres": 12.0, "scales": 30.0}.get(name, 5.0))
    rays = np.concatenate([rays, np.array([[np.nan, 0, 0, 0, 0, 1], [np.inf, 0, 0, 1, 0, 0], [1e31, 0, 0, -1, 0, 0]], F32)])
    want, visits = r.trace_rays(rays)
    got, _ = r.trace_rays(rays, with_visits=False)
    # a bounce: from the hit points, where the nearest surface is at t = 0
    k = want["hit"] == 1
    hp = rays[k, :3] + want["t"][k, None] * rays[k, 3:]
    again = np.concatenate([hp, -rays[k, 3:] + np.random.default_rng(1).normal(size=hp.shape)], 1).astype(F32)
    want2, _ = r.trace_rays(again)
    got2, _ = r.trace_rays(again, with_visits=False)
    r.close()
    assert np.array_equal(want.view(np.uint32), got.view(np.uint32))
    assert np.array_equal(want2.view(np.uint32), got2.view(np.uint32))
    assert visits.max() > 0


def _progress(r, state, camera, kernel, counting):
    r.set_resolution(67, 41)
    state.kernel = kernel
    r.set_state(state.to_struct())
    r.set_camera(camera.to_struct())
    r.enable_counters(counting)
    r.render()
    acc, rng, _ = r.progress()
    return acc.view(np.uint32), rng, r.framebuffer().view(np.uint32)


@pytest.mark.parametrize("semantics", [_lib.SEMANTICS_HIP, _lib.SEMANTICS_WGSL], ids=["hip", "wgsl"])
@pytest.mark.parametrize("kernel", [_lib.KERNEL_MEGA, _lib.KERNEL_WAVEFRONT], ids=["mega", "wavefront"])
@pytest.mark.parametrize("name", ["copies", "slivers", "mixed", "room", "instanced"])
def test_pictures_equal_the_reference_walks(name, kernel, semantics):
    scene = SCENES[name]()
    r = ornament.Renderer(ornament.Bvh(scene), device=0)
    state = ornament.State()
    state.setDepth(8)
    state.setIterations(6)
    state.setGamma(2.2)
    state.semantics = semantics
    want = _progress(r, state, scene.camera, _lib.KERNEL_MEGA, True)
    got = _progress(r, state, scene.camera, kernel, False)
    r.close()
    for a, b in zip(want, got):
        assert np.array_equal(a, b)


def test_blobs_with_other_boxes_keep_the_reference_walk():
    """A leaf box wider than its triangle, and a child box outside its
    parent's: such blobs are taken as before, and walked the reference's way."""
    scene = SCENES["mixed"]()
    for change in ("wide_leaf", "child_outside"):
        bvh = ornament.Bvh(scene)
        inner = np.nonzero(bvh.blas_nodes["node_type"] == 0)[0]
        if change == "wide_leaf":
            kinds = bvh.blas_nodes["node_type"][bvh.blas_nodes["left_or_custom_id"][inner]]
            i = inner[kinds == 3][0]
            bvh.blas_nodes["left_aabb_min_or_v0"][i] -= 0.05
        else:
            bvh.blas_nodes["left_aabb_max_or_v1"][inner[-1]] -= 0.2
        r = ornament.Renderer(bvh, device=0)
        rays = _rays(5.0, 20_000)
        want, _ = r.trace_rays(rays)
        got, _ = r.trace_rays(rays, with_visits=False)
        r.close()
        assert np.array_equal(want.view(np.uint32), got.view(np.uint32))


@pytest.mark.parametrize("builder", ["reference", "sah", "lbvh"])
@pytest.mark.parametrize("semantics", [_lib.SEMANTICS_HIP, _lib.SEMANTICS_WGSL], ids=["hip", "wgsl"])
def test_large_scenes_render_the_same_on_any_tree_rule(builder, semantics):
    """Past 16384 nodes the trees' areas decide what a plain render walks; a
    counting render always walks the blob's."""
    w, h = 97, 53
    scene = scenes.instanced_meshes_scene(w, h, seed=3, n_blas=2, n_instances=24, tri_range=(8_000, 12_000),
                                          texture_size=32)
    bvh = ornament.Bvh(scene, builder=builder)
    frames = []
    for count in (False, True):
        pt = ornament.PathTracer(scene, bvh=bvh)
        scene.camera.dirty = True
        pt.state.setDepth(8)
        pt.state.setIterations(3)
        pt.state.semantics = semantics
        pt.setResolution(ornament.Resolution(w, h))
        pt.renderer.enable_counters(count)
        pt.render()
        frames.append(pt.getFrameBuffer().copy())
        pt.deinit()
    assert np.array_equal(frames[0].view(np.uint32), frames[1].view(np.uint32))
