"""Signs of a closed mesh on rows of samples that run exactly through the shared
edges and corners of its triangles, at coordinates whose differences and products
are not exact in any floating-point format: every sample has the oracle's sign."""
import numpy as np
import pytest

from oracle import meshsdf_oracle as mso
from test_meshsdf import cube_mesh, icosphere

pytestmark = pytest.mark.gpu


def cube(lo, hi):
    v, t = cube_mesh()
    return np.where(v < 0, np.float32(lo), np.float32(hi)).astype(np.float32), t


def lathe():
    """A closed body of revolution about z; sin(pi) leaves coordinates near 1e-16."""
    m, rings = 16, [(0.5, -0.75), (1.0, 0.0), (0.5, 0.75)]
    v = [[r * np.cos(2 * np.pi * a / m), r * np.sin(2 * np.pi * a / m), z]
         for r, z in rings for a in range(m)] + [[0, 0, -1.25], [0, 0, 1.25]]
    t = []
    for a in range(m):
        b = (a + 1) % m
        t.append((len(v) - 2, b, a))
        for k in range(len(rings) - 1):
            p, q, r, s = k * m + a, k * m + b, (k + 1) * m + a, (k + 1) * m + b
            t += [(p, q, s), (p, s, r)]
        top = (len(rings) - 1) * m
        t.append((len(v) - 1, top + a, top + b))
    return np.array(v, np.float32), np.array(t, np.int32)


def cases():
    for lo, hi, dx, pad in [(0.1, 1.1, 0.05, 2), (0.01, 1.01, 0.05, 2), (0.001, 0.7, 0.02, 2),
                            (-0.7, 1.3, 0.05, 3)]:
        yield f"cube_{lo}_{hi}", *cube(lo, hi), dx, pad
    yield "lathe", *lathe(), 0.125, 2
    yield "sphere", *icosphere(2), 0.1, 2


@pytest.mark.parametrize("case", list(cases()), ids=lambda c: c[0])
def test_every_sign(case):
    from sphpc_b200 import meshsdf
    _, v, t, dx, pad = case
    dims, origin = meshsdf.sdfgen_grid(v, dx, pad)
    got = meshsdf.mesh_sdf(v, t, dims, origin, dx).astype(np.float64)
    want = mso.grid_sdf(v, t, dims, origin, dx)
    # FP32 distances within 3 of the origin
    assert np.max(np.abs(np.abs(got) - np.abs(want))) < 2e-6
    # samples within the rounding of their FP32 coordinates may lie on either side
    off = np.abs(want) > 1e-6
    assert np.array_equal(np.sign(got[off]), np.sign(want[off]))
