"""Mesh distance fields where the sign or the culling can go wrong: rows of
samples through edges and corners, corners that are not shared by index, two
nested shells, a mesh with a hole or a flipped triangle (fractional winding
numbers), fewer triangles than a cluster, samples far outside."""
import numpy as np
import pytest

from oracle import meshsdf_oracle as mso
from test_meshsdf import cube_mesh, icosphere

pytestmark = pytest.mark.gpu


def unwelded(v, t):
    return v[t].reshape(-1, 3), np.arange(3 * len(t), dtype=np.int32).reshape(-1, 3)


def shells():
    v, t = icosphere(2, 1.0)
    w, u = icosphere(1, 0.4)
    return np.concatenate([v, w]), np.concatenate([t, u[:, ::-1] + len(v)])


def cases():
    v, t = icosphere(2)
    flipped = t.copy()
    flipped[17] = flipped[17][::-1]
    yield "cube_on_rows", *cube_mesh(), (9, 9, 9), (-2.0, -2.0, -2.0), 0.5
    yield "sphere_on_rows", v, t, (9, 9, 9), (-1.0, -1.0, -1.0), 0.25
    yield "unwelded", *unwelded(v, t), (9, 7, 8), (-1.9, -1.6, -1.7), 0.45
    yield "shells", *shells(), (11, 10, 9), (-1.2, -1.1, -1.0), 0.23
    yield "hole", v, t[5:], (9, 7, 8), (-1.9, -1.6, -1.7), 0.45
    yield "flipped", v, flipped, (9, 7, 8), (-1.9, -1.6, -1.7), 0.45
    yield "tetrahedron", np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], np.float32), \
        np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], np.int32), (5, 6, 7), \
        (-0.31, -0.27, -0.19), 0.21
    yield "far", v, t, (5, 3, 3), (30.0, -1.0, -1.0), 7.0
    yield "one_sample", v, t, (1, 1, 1), (0.1, 0.2, 0.3), 1.0


@pytest.mark.parametrize("case", list(cases()), ids=lambda c: c[0])
def test_mesh_sdf_edges(case):
    from sphpc_b200 import meshsdf
    _, v, t, dims, origin, dx = case
    got = meshsdf.mesh_sdf(v, t, dims, origin, dx).astype(np.float64)
    want = mso.grid_sdf(v, t, dims, origin, dx)
    # FP32 distances of points within 60 of the origin: a few ulp of that
    assert np.max(np.abs(np.abs(got) - np.abs(want))) < 2e-6 * max(1.0, np.abs(want).max())
    off = np.abs(want) > 1e-3
    assert np.array_equal(np.sign(got[off]), np.sign(want[off]))
