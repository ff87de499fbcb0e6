"""GPU-built linear BVHs at the limits of their inputs."""
import numpy as np
import pytest

from zig_ornament_gb300 import ornament

pytestmark = pytest.mark.gpu


def _leaves(bvh):
    """Triangles of a single mesh's tree from left to right."""
    nodes, out, todo = bvh.blas_nodes, [], [len(bvh.blas_nodes) - 1]
    while todo:
        n = nodes[todo.pop()]
        if n["node_type"] == 3:
            out.append(int(n["left_or_custom_id"]))
        else:
            todo += [n["right_or_material_index"], n["left_or_custom_id"]]
    return np.array(out)


def _codes(v):
    """Morton codes within the bounds of the centres, in single precision; a centre
    is of the least and the largest coordinate by `<` from the first vertex on."""
    with np.errstate(invalid="ignore"):
        mn, mx = v[:, 0].copy(), v[:, 0].copy()
        for j in (1, 2):
            mn, mx = np.where(v[:, j] < mn, v[:, j], mn), np.where(v[:, j] > mx, v[:, j], mx)
        bounds = np.float32(0.5) * (mn + mx)
        lo, hi = np.nanmin(bounds, 0), np.nanmax(bounds, 0)
        c = np.float32(0.5) * (np.fmin.reduce(v, 1) + np.fmax.reduce(v, 1))
        f = np.clip((c - lo) * (np.float32(1023) / (hi - lo)), 0, 1023).astype(np.uint32)
    return sum(((f[:, k] >> b) & 1) << (3 * b + 2 - k) for k in range(3) for b in range(10))


@pytest.mark.parametrize("vertex", [None, 0, 1, 2])
def test_nan_vertices_and_the_bounds_of_the_codes(vertex):
    rs = np.random.default_rng(3)
    v = (rs.uniform(-1, 1, (700, 1, 3)) + rs.uniform(-0.05, 0.05, (700, 3, 3))).astype(np.float32)
    if vertex is not None:
        v[[5, 300]] += np.float32(40.0)   # what is left of these is far away
        v[[5, 300], vertex] = np.nan
    s = ornament.Scene()
    idx = np.arange(2100, dtype=np.uint32)
    flat = np.concatenate([v.reshape(-1, 3), np.ones((2100, 1), np.float32)], 1).astype(np.float32)
    n = np.tile(np.array([0, 1, 0, 0], np.float32), (2100, 1))
    m = s.createMesh(flat, idx, n, idx, np.zeros((0, 2), np.float32), np.zeros(0, np.uint32), ornament.identity(),
                     s.lambertian((0.5, 0.5, 0.5, 1.0)))
    m.aabb = ornament.Aabb(np.array([-2, -2, -2, 1], np.float32), np.array([50, 50, 50, 1], np.float32))   # (has to be finite)
    s.attachMesh(m)
    got = _leaves(ornament.Bvh(s, builder="lbvh"))
    code = _codes(v)
    assert np.array_equal(got, np.lexsort((np.arange(700), code)))
