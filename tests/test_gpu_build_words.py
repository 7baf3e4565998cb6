"""Neighbour build: rows of more than 32 candidates (several hit words a row), more
hit words than a thread's column holds, and the cap of 60, with and without a
tile, equal the oracle's buckets bit for bit; and the FP32 pre-test's band, as
wide as the grid needs, decides no pair wrongly."""
import numpy as np
import pytest

from helpers import oracle_for
from sphpc_b200 import Simulation, _lib
from sphpc_b200.scenes import config_path


def scene(tmp_path, dims):
    text = open(config_path("small_dam")).read()
    text = text.replace("number_particles = 4096", f"number_particles = {dims[0] * dims[1] * dims[2]}")
    for axis, m, old_box in zip("xyz", dims, (48.0, 24.0, 24.0)):
        text = text.replace(f"max_{axis} = {old_box}", f"max_{axis} = {3.0 * m:.9g}")
        text = text.replace(f"max_{axis} = 16.0", f"max_{axis} = {float(m):.9g}")
    path = tmp_path / "scene.ini"
    path.write_text(text)
    return Simulation(str(path))


@pytest.mark.gpu
@pytest.mark.parametrize("dims,scale", [
    ((11, 11, 11), (0.8, 0.8, 0.8)),     # one tile; rows of about 47
    ((11, 11, 11), (0.5, 0.5, 0.5)),     # one tile; rows of about 190, the cap
    ((11, 11, 11), (0.1, 0.1, 0.1)),     # one tile; all in one cell or two
    ((90, 4, 4), (0.25, 1.0, 1.0)),      # one tile; long thin rows
    ((4, 4, 90), (1.0, 1.0, 0.25)),      # one tile; many short rows
    ((90, 5, 4), (0.2, 1.5, 1.5)),       # no tile; rows of about 40, few hits each
    ((31, 31, 31), (0.4, 1.3, 1.3)),     # no tile in the middle
    # the room of a tile by the blocks an SM: 4056, 3552, 2344 and 1744 records
    ((15, 16, 16), (0.45, 0.45, 0.45)),
    ((15, 16, 16), (0.6, 0.6, 0.6)),
    ((26, 26, 26), (0.62, 0.62, 0.62)),
    ((38, 38, 38), (0.7, 0.7, 0.7)),
    ((42, 42, 42), (0.85, 0.85, 0.85)),
])
def test_buckets_of_dense_rows(tmp_path, dims, scale):
    with scene(tmp_path, dims) as sim:
        rng = np.random.default_rng(11)
        pos = {}
        for f, s in zip(("x", "y", "z"), scale):
            x = s * (sim.host(f).copy() + 0.3 * rng.uniform(-1, 1, sim.n)) + 0.5
            pos[f] = x.astype(np.float32).astype(np.float64)
        pos.update({f + "_star": v for f, v in pos.items()})
        sim.push(pos)
        sim.find_all_neighbors()
        o = oracle_for(sim, sim.fetch())
        o.call("find_all_neighbors")
        cnt, nbr = sim.neighbor_buckets()
        ocnt, onbr = o.neighbor_lists()
        np.testing.assert_array_equal(cnt, ocnt)
        used = np.arange(nbr.shape[1])[None, :] < cnt[:, None]
        np.testing.assert_array_equal(np.where(used, nbr, 0), np.where(used, onbr, 0))
        assert sim.device_errors() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.05, 0.2])
def test_crowded_cells_keep_their_order(tmp_path, scale):
    """4913 particles in one cell (and in eight): the slots by counting and, once
    the host has seen the crowded cell, by digit passes are the oracle's."""
    with scene(tmp_path, (17, 17, 17)) as sim:
        rng = np.random.default_rng(3)
        pos = {f: (scale * rng.permutation(sim.host(f)) + 0.1).astype(np.float32).astype(np.float64)
               for f in ("x", "y", "z")}
        pos.update({f + "_star": v for f, v in pos.items()})
        sim.push(pos)
        o = oracle_for(sim, sim.fetch())
        o.call("find_all_neighbors")
        ocnt, onbr = o.neighbor_lists()
        for _ in range(3):
            sim.find_all_neighbors()
            cnt, nbr = sim.neighbor_buckets()
            np.testing.assert_array_equal(cnt, ocnt)
            used = np.arange(nbr.shape[1])[None, :] < cnt[:, None]
            np.testing.assert_array_equal(np.where(used, nbr, 0), np.where(used, onbr, 0))
        assert sim.device_errors() == 0


@pytest.mark.parametrize("h", [2.0, 1.0, 0.0125, 3.0])
@pytest.mark.parametrize("cells", [1, 37, 128, 384, 768, 2000])
def test_band_covers_the_rounding_of_its_grid(h, cells):
    m = h * cells
    band = _lib.load().sphpc_neighbor_pretest_band(m, h)
    assert 0.0 < band <= 1.12 * 2.0 ** -10 * h * h
    f = np.float32
    rng = np.random.default_rng(cells)
    n = 400_000
    xp = m * (1.0 - 0.5 ** (1 + 20 * rng.random((n, 3))))
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    xq = xp + u * (h * (1.0 + (rng.random(n) - 0.5) * 4.0 * band / (h * h)))[:, None]
    exact = np.sum((xp - xq) ** 2, axis=1) < h * h
    # s = r^2 - h^2 by fused multiply-adds from -h^2, as the tiles are tested
    d = (xp.astype(f) - xq.astype(f)).astype(np.float64)
    s = np.full(n, -f(h * h), dtype=f)
    for k in range(3):
        s = (d[:, k].astype(f).astype(np.float64) ** 2 + s.astype(np.float64)).astype(f)
    b = f(band)
    assert not np.any((s < -b) & ~exact)
    assert not np.any((s > b) & exact)
    assert np.any(np.abs(s) <= b) and np.any(s > b) and np.any(s < -b)
