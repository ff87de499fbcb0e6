"""The near-first walk at the limits of what makes its results the reference
walk's: closest hits bit for bit those of the walk that counts visits."""
import numpy as np
import pytest

from zig_ornament_gb300 import ornament, scenes
from zig_ornament_gb300.ornament import F32, identity, mul, scaling, translation

pytestmark = pytest.mark.gpu


def _rays(extent, n=200_000, seed=11):
    rs = np.random.default_rng(seed)
    o, d = rs.uniform(-extent, extent, (n, 3)), rs.normal(size=(n, 3))
    k, row = n // 8, np.arange(n // 8)
    d[row, rs.integers(0, 3, k)] *= 10.0 ** rs.uniform(-7, -1, k)    # nearly along a box's faces
    d[k:2 * k] = -o[k:2 * k]                                         # towards the middle
    d[2 * k:3 * k] = 0.0                                             # along an axis
    d[2 * k + row, rs.integers(0, 3, k)] = rs.choice([-1.0, 1.0], k)
    d[3 * k:4 * k] *= 10.0 ** rs.uniform(-6, 6, (k, 1))              # directions of any length
    return np.concatenate([o, d], 1).astype(F32)


def _assert_same_hits(scene, extent, epsilon=0.001, trees=True, middle=0.0):
    """Rays in a cube about `middle`, and a bounce from what they hit."""
    r = ornament.Renderer(ornament.Bvh(scene), device=0)
    state = ornament.State()
    state.setRayCastEpsilon(epsilon)
    r.set_state(state.to_struct())
    assert (r.near_trees() > 0) == trees
    rays = _rays(extent)
    rays[:, :3] += F32(middle)
    hit = 0
    for _ in range(2):
        want, _ = r.trace_rays(rays)
        got, _ = r.trace_rays(rays, with_visits=False)
        assert np.array_equal(want.view(np.uint32), got.view(np.uint32))
        k = (want["hit"] == 1) & np.isfinite(want["t"])
        hit += np.count_nonzero(k)
        hp = rays[k, :3] + want["t"][k, None] * rays[k, 3:]
        rays = np.concatenate([hp, np.random.default_rng(2).normal(size=hp.shape)], 1).astype(F32)
    r.close()
    assert hit > 10_000


def test_negative_radii():
    """A hollow ball is a sphere of negative radius: its box's corners change places."""
    s = ornament.Scene()
    rs = np.random.default_rng(0)
    grey = s.lambertian((0.5, 0.5, 0.5, 1.0))
    for i in range(30):
        r = rs.uniform(0.3, 1.2)
        s.createSphere((*rs.uniform(-4, 4, 3), 1), -r if i % 3 == 0 else r, grey)
    _assert_same_hits(s, 5.0, trees=False)


@pytest.mark.parametrize("epsilon,trees", [(1.0, True), (-0.001, False), (-5.0, False), (float("nan"), False)])
def test_ray_cast_epsilon(epsilon, trees):
    """The near-first trees are walked for hits from the origin on, not for hits behind it."""
    _assert_same_hits(scenes.spheres_scene(), 12.0, epsilon, trees)


def test_epsilon_zero():
    """Rays that start on a surface hit it at t = 0, and its neighbour's box lies beyond."""
    _assert_same_hits(scenes.spheres_scene(), 12.0, 0.0)


def _terrain(offset, cell, n=16, sheets=2, seed=0):
    """Sheets of n x n cells of two triangles, about `offset`."""
    rs = np.random.default_rng(seed)
    tris = []
    for k in range(sheets):
        g = np.arange(n + 1) - n / 2
        h = rs.uniform(-0.6, 0.6, (n + 1, n + 1)) * cell - 1.5 * k * cell
        p = np.stack(np.broadcast_arrays(g[:, None] * cell, h, g[None, :] * cell), -1) + offset
        a, b, c, d = p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]
        tris += [np.stack([a, b, c], 2).reshape(-1, 3, 3), np.stack([a, c, d], 2).reshape(-1, 3, 3)]
    return np.concatenate(tris)


def _terrains(offset, cell, extent, scales=(1.0,), instances=40, world=0.0):
    """A mesh modelled `offset` away from its origin, and instances that bring it back."""
    s = ornament.Scene()
    rs = np.random.default_rng(1)
    o = np.array([offset, 0.5 * offset, -offset])
    v = np.concatenate([_terrain(o, cell).reshape(-1, 3), np.ones((3 * 1024, 1))], 1).astype(F32)
    idx = np.arange(len(v), dtype=np.uint32)
    n = np.tile(np.array([0, 1, 0, 0], F32), (len(v), 1))
    back = translation(*-o)
    m = s.createMesh(v, idx, n, idx, np.zeros((0, 2), F32), np.zeros(0, np.uint32), mul(back, translation(*[world] * 3)),
                     s.lambertian((0.5, 0.5, 0.5, 1.0)))
    for _ in range(instances):
        turn = identity()
        turn[:3, :3] = np.linalg.qr(rs.normal(size=(3, 3)))[0]
        size = scaling(*[float(rs.choice(scales) * rs.uniform(0.5, 1.5))] * 3)
        at = translation(*(world + rs.uniform(-0.8, 0.8, 3) * extent))
        s.createMeshInstance(m, mul(mul(mul(back, turn), size), at).astype(F32), s.materials[0])
    return s


@pytest.mark.parametrize("offset,cell", [(0.0, 0.25), (1e4, 0.25), (1e5, 0.02), (1e5, 0.25), (1e6, 1.0), (1e7, 4.0)])
def test_meshes_far_from_their_own_origin(offset, cell):
    """Survey and city data: the rounding of a mesh's own coordinates is larger
    than the detail of the scene that its transforms bring it back to."""
    extent = 16 * cell
    _assert_same_hits(_terrains(offset, cell, extent), extent)


@pytest.mark.parametrize("world", [1e3, 1e5])
def test_scenes_far_from_the_origin(world):
    _assert_same_hits(_terrains(0.0, 0.25, 4.0, world=world), 4.0, middle=world)


def test_instances_of_many_sizes():
    _assert_same_hits(_terrains(300.0, 0.25, 6.0, scales=(0.01, 0.1, 1.0, 10.0)), 6.0)


@pytest.mark.parametrize("change,trees", [("shrunk", False), ("moved", False), ("grown", True)])
def test_boxes_of_shapes_as_a_caller_gives_them(change, trees):
    """The boxes of shapes come from the caller, who can give any: with one that does
    not hold its shape, what a ray hits depends on the order of its visits."""
    s = _terrains(0.0, 0.25, 4.0)
    rs = np.random.default_rng(4)
    for shape in s.mesh_instances + s.meshes:
        lo, hi = shape.aabb.min.copy(), shape.aabb.max.copy()
        e = hi - lo
        if change == "shrunk":
            lo, hi = lo + F32(0.3) * e, hi - F32(0.3) * e
        elif change == "moved":
            by = rs.uniform(-0.7, 0.7, 4).astype(F32) * e
            lo, hi = lo + by, hi + by
        else:
            lo, hi = lo - e, hi + e
        shape.aabb = ornament.Aabb(lo, hi)
    _assert_same_hits(s, 4.0, trees=trees)


def test_rays_from_far_away():
    r = ornament.Renderer(ornament.Bvh(_terrains(0.0, 0.25, 4.0)), device=0)
    rs = np.random.default_rng(8)
    o = rs.uniform(-4, 4, (200_000, 3)) * 10.0 ** rs.uniform(0, 6, (200_000, 1))
    rays = np.concatenate([o, rs.uniform(-3, 3, o.shape) - o], 1).astype(F32)
    want, _ = r.trace_rays(rays)
    got, _ = r.trace_rays(rays, with_visits=False)
    r.close()
    assert np.array_equal(want.view(np.uint32), got.view(np.uint32))
    assert np.count_nonzero(want["hit"]) > 10_000
