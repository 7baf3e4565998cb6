"""Particles beyond a grid that is one cell wide along an axis (a flat box): they are
reported, and every bucket is that of the 27-cell walk over the cell table."""
import numpy as np
import pytest

from sphpc_b200 import Simulation
from sphpc_b200.scenes import config_path

pytestmark = pytest.mark.gpu
CELL_RANGE = 1 << 2


def walk(x, h, dims, ids, start):
    """Buckets by particle, 60 at most."""
    out = []
    for p, xp in enumerate(x):
        found = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    s = xp + h * np.array([dx, dy, dz])
                    c = np.floor(s / h)
                    if np.any(s < 0) or np.any(c > np.array(dims) - 1):
                        continue
                    c = c.astype(int)
                    key = c[0] + dims[0] * (c[1] + dims[1] * c[2])
                    q = ids[start[key]:start[key + 1]]
                    q = q[q != p]
                    d = xp - x[q]
                    found += list(q[(d * d) @ np.ones(3) < h * h])
        out.append(found[:60])
    return out


@pytest.mark.parametrize("axis", ["y", "z"])
@pytest.mark.parametrize("offset", [0.0, 10.0])
def test_flat_box(tmp_path, axis, offset):
    text = open(config_path("small_dam")).read().replace("number_particles = 4096",
                                                         "number_particles = 700")
    for f, old in zip("xyz", (48.0, 24.0, 24.0)):
        size = 0.0 if f == axis else 30.0
        text = text.replace(f"max_{f} = {old}", f"max_{f} = {size}")
    path = tmp_path / "flat.ini"
    path.write_text(text)
    with Simulation(str(path)) as sim:
        h, n = sim.params.smoothing_radius, sim.n
        dims = (sim.neighbors.hash_size_x, sim.neighbors.hash_size_y, sim.neighbors.hash_size_z)
        assert dims["xyz".index(axis)] == 1
        rng = np.random.default_rng(4)
        # multiples of 2^-10: every distance is exact
        x = np.round(rng.uniform(0.0, 12.0, (n, 3)) * 1024) / 1024
        x[:, "xyz".index(axis)] = offset + np.round(rng.uniform(0, 2.9 * h, n) * 1024) / 1024
        pos = {f: x[:, k].copy() for k, f in enumerate("xyz")}
        pos.update({f + "_star": v for f, v in pos.items()})
        sim.push(pos)
        sim.find_all_neighbors()
        cnt, nbr = sim.neighbor_buckets()
        _, ids, start = sim.cell_data()
        want = walk(x, h, dims, ids, start)
        assert [int(c) for c in cnt] == [len(w) for w in want]
        for p, w in enumerate(want):
            assert [int(q) for q in nbr[p, :cnt[p]]] == [int(q) for q in w]
        assert sim.device_errors() == CELL_RANGE
