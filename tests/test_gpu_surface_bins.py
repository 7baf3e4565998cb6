"""Particle surface: distances over bins and smoothing by tiles against the
definition in FP64, on grids whose sides are no multiples of the blocks, with
particles outside the grid, many particles in a bin, long reaches and empty
parts.

Tolerance: coordinates up to 32 are rounded to FP32 within 2^-20 (particle and
voxel, 1.9e-6 each, and their difference), so a distance is off by less than
sqrt(3) 6e-6; the fixed point adds 2^-21 and nine means 9 x 3e-7 of values below
9: together below 2e-5."""
import numpy as np
import pytest

from sphpc_b200.surface import particle_surface


def definition(xyz, radius, half_width, dims, origin):
    voxel = radius / 2.0
    band = half_width * voxel + radius
    nx, ny, nz = dims
    ax = [np.arange(m) * voxel + o for m, o in zip(dims, origin)]
    g = np.stack(np.meshgrid(*ax, indexing="ij"), axis=-1).reshape(-1, 3)
    best = np.full(len(g), np.inf)
    for q in np.array_split(xyz, max(1, len(xyz) // 200)):
        best = np.minimum(best, ((g[:, None, :] - q[None]) ** 2).sum(-1).min(1))
    phi = np.clip(np.sqrt(best) - radius, -band, band).reshape(nx, ny, nz) - radius
    for _ in range(3):
        for axis in range(3):
            p = np.concatenate([phi.take([0], axis), phi, phi.take([-1], axis)], axis)
            m = phi.shape[axis]
            phi = (p.take(range(m), axis) + phi + p.take(range(2, m + 2), axis)) / 3.0
    return (phi + radius).transpose(2, 1, 0).reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,n,radius,half_width,spread", [
    ((33, 9, 17), 300, 1.0, 2, 1.0),     # one past the tiles
    ((31, 8, 7), 60, 1.0, 2, 1.6),       # particles outside the grid
    ((1, 1, 40), 20, 1.0, 2, 1.0),       # a line of voxels
    ((5, 38, 3), 1, 1.0, 2, 1.0),        # one particle, most voxels out of reach
    ((20, 21, 22), 900, 1.0, 2, 0.15),   # bins of many
    ((24, 20, 18), 40, 1.0, 9, 1.2),     # a long reach: wider bins
    ((26, 27, 12), 200, 0.37, 1, 1.0),   # a radius that is no power of two
])
def test_surface_matches_definition(dims, n, radius, half_width, spread):
    rng = np.random.default_rng(n)
    size = (np.array(dims) - 1) * radius / 2.0
    origin = (-3.0, 2.0, 0.25)
    mid = np.array(origin) + size / 2.0
    xyz = mid + spread * (size + 1.0) * (rng.random((n, 3)) - 0.5)
    got = particle_surface(xyz, radius, half_width, dims, origin)[0]
    want = definition(xyz, radius, half_width, dims, origin)
    np.testing.assert_allclose(got, want, rtol=0.0, atol=2e-5)
