"""Cells of many particles: the counted slots of cells on both sides of the line
between ranking by comparing and ordering by one block, in sets whose ids take two
and four digit passes; a step that first crowds takes time in proportion to its
particles; and a set that spreads out again is counted again."""
import numpy as np
import pytest

from sphpc_b200 import Simulation
from sphpc_b200.scenes import config_path

pytestmark = pytest.mark.gpu


def scene(tmp_path, dims):
    text = open(config_path("small_dam")).read()
    text = text.replace("number_particles = 4096", f"number_particles = {dims[0] * dims[1] * dims[2]}")
    for axis, m, old_box in zip("xyz", dims, (48.0, 24.0, 24.0)):
        text = text.replace(f"max_{axis} = {old_box}", f"max_{axis} = {3.0 * m:.9g}")
        text = text.replace(f"max_{axis} = 16.0", f"max_{axis} = {float(m):.9g}")
    path = tmp_path / "scene.ini"
    path.write_text(text)
    return Simulation(str(path))


def crowd(sim, sizes, rng):
    """Particles in any order of their ids: `sizes` of them in one cell each (every
    other cell along x, y and z, h = 2), the rest where the scene has them."""
    pos = {f: sim.host(f).copy() for f in ("x", "y", "z")}
    who = rng.permutation(sim.n)
    at = 0
    for k, m in enumerate(sizes):
        cell = np.array([2 * (k % 3), 2 * (k // 3 % 3), 2 * (k // 9)])
        for f, c in zip(("x", "y", "z"), cell):
            pos[f][who[at:at + m]] = 2.0 * c + rng.uniform(0.1, 1.9, m)
        at += m
    pos = {f: v.astype(np.float32).astype(np.float64) for f, v in pos.items()}
    pos.update({f + "_star": v for f, v in pos.items()})
    sim.push(pos)
    return pos


def check_slots(sim, pos):
    keys, ids, start = sim.cell_data()
    nx, ny = sim.neighbors.hash_size_x, sim.neighbors.hash_size_y
    c = [np.floor(pos[f] / 2.0).astype(np.int64) for f in ("x", "y", "z")]
    key = c[0] + nx * (c[1] + ny * c[2])
    want = np.argsort(key, kind="stable")
    np.testing.assert_array_equal(ids, want)
    np.testing.assert_array_equal(keys, key[want])
    np.testing.assert_array_equal(start, np.searchsorted(key[want], np.arange(len(start))))
    assert sim.device_errors() == 0


@pytest.mark.parametrize("dims,sizes", [
    ((16, 16, 16), (512, 513, 514, 700, 1)),
    ((16, 16, 16), (4096,)),
    ((64, 32, 32), (2047, 2048, 2049, 4097, 513, 512, 511, 2300, 6000)),      # 65,536
    ((41, 41, 39), (2047, 2049, 4096, 513, 513, 513, 513, 513, 513, 9000)),   # 65,559
    ((70, 50, 20), (513,) * 18 + (20_000,)),
])
def test_slots_of_crowded_cells(tmp_path, dims, sizes):
    with scene(tmp_path, dims) as sim:
        rng = np.random.default_rng(len(sizes))
        pos = crowd(sim, sizes, rng)
        for _ in range(3):   # counted, then by digit passes
            sim.find_all_neighbors()
            check_slots(sim, pos)


def slot_times(sim, searches=1):
    sim.profile(True)
    for _ in range(searches):
        sim.find_all_neighbors()
    times = sim.profile_read()
    sim.profile(False)
    return times


def test_first_crowded_search_is_linear(tmp_path):
    """1,048,576 particles in one cell: one block puts them in order, about 3 ns a
    particle and digit pass, 14 ms.  Comparing each with all took 12.7 ms for
    262,144, so it would take 200."""
    with scene(tmp_path, (128, 128, 64)) as sim:
        slot_times(sim, 3)
        pos = crowd(sim, (sim.n,), np.random.default_rng(7))
        times = slot_times(sim)
        assert "count_cells" in times
        assert times["count_cells"][1] + times["reorder"][1] < 40.0
        check_slots(sim, pos)


def test_a_set_that_spreads_out_is_counted_again(tmp_path):
    with scene(tmp_path, (16, 16, 16)) as sim:
        home = {f: sim.host(f).copy() for f in ("x", "y", "z")}
        home.update({f + "_star": v for f, v in home.items()})
        crowd(sim, (1000,), np.random.default_rng(9))
        slot_times(sim, 2)
        assert "radix_sort" in slot_times(sim)
        sim.push(home)
        times = slot_times(sim, 200)
        assert times["count_cells"][0] > 100
        check_slots(sim, home)
