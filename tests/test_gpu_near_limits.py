"""The near-first walk at the limits of what makes its results the reference
walk's: closest hits bit for bit those of the walk that counts visits."""
import numpy as np
import pytest

from zig_ornament_gb300 import ornament, scenes
from zig_ornament_gb300.ornament import F32

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


def _assert_same_hits(scene, extent, epsilon=0.001, trees=2, middle=0.0):
    """Rays in a cube about `middle`, and a bounce from what they hit."""
    r = ornament.Renderer(ornament.Bvh(scene), device=0)
    state = ornament.State()
    state.setRayCastEpsilon(epsilon)
    r.set_state(state.to_struct())
    assert r.near_trees() == trees
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
    _assert_same_hits(s, 5.0, trees=0)


@pytest.mark.parametrize("epsilon,trees", [(1.0, 2), (-0.001, 0), (-5.0, 0), (float("nan"), 0)])
def test_ray_cast_epsilon(epsilon, trees):
    """The near-first trees are walked for hits from the origin on, not for hits behind it."""
    _assert_same_hits(scenes.spheres_scene(), 12.0, epsilon, trees)
