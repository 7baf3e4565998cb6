"""Neighbour lists with tiles: the buckets
equal the oracle's bit for bit where the tiles' edges lie -- odd counts, blocks
over the end of a row of cells, a smoothing radius that is no power of two,
cells of many particles (tiles that do not fit, the 60-neighbour cap) and of
few -- and one fused step on them stays within the one-step parity bounds."""
import numpy as np
import pytest

from helpers import assert_close, oracle_for, oracle_state
from sphpc_b200 import Simulation
from sphpc_b200.scenes import config_path

pytestmark = pytest.mark.gpu


def scene(tmp_path, dims, spacing=1.0, box=(3.0, 2.0, 1.5)):
    text = open(config_path("small_dam")).read()
    n = dims[0] * dims[1] * dims[2]
    text = text.replace("number_particles = 4096", f"number_particles = {n}")
    for axis, (m, f, old_box) in zip("xyz", zip(dims, box, (48.0, 24.0, 24.0))):
        size = m * spacing
        text = text.replace(f"max_{axis} = {old_box}", f"max_{axis} = {f * size:.9g}")
        text = text.replace(f"max_{axis} = 16.0", f"max_{axis} = {size:.9g}")
    path = tmp_path / "scene.ini"
    path.write_text(text)
    return Simulation(str(path))


@pytest.mark.parametrize("dims,spacing,scale,noise", [
    ((41, 43, 41), 1.0, 1.0, 0.2),      # 72,283: an odd count, a last block of 91
    ((5, 5, 5), 1.0, 1.0, 0.2),         # one block, not full
    ((3, 43, 1), 1.0, 1.0, 0.2),        # 129: a block of one
    ((127, 33, 17), 1.0, 1.0, 0.4),     # long rows, few planes
    ((17, 68, 68), 0.83, 1.0, 0.3),     # short rows: most blocks run over a row's end
    ((41, 41, 41), 1.0, 0.72, 0.3),     # 21 particles a cell: some tiles do not fit
    ((41, 41, 41), 1.0, 0.45, 0.3),     # 90 a cell: the cap, no tile fits
    ((41, 41, 41), 1.0, 1.45, 0.5),     # 2.6 a cell
])
def test_tiled_buckets_bit_exact(tmp_path, dims, spacing, scale, noise):
    with scene(tmp_path, dims, spacing) as sim:
        rng = np.random.default_rng(7)
        pos = {}
        for f in ("x", "y", "z"):
            x = sim.host(f).copy()
            x = x * scale + spacing * noise * rng.uniform(-1, 1, sim.n)
            pos[f] = np.clip(x, 1e-3, None).astype(np.float32).astype(np.float64)
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


def test_tiled_step_matches_oracle(tmp_path):
    with scene(tmp_path, (41, 43, 41)) as sim:
        sim.step(3)
        o = oracle_for(sim, sim.fetch())
        sim.step(1)
        o.step(1)
        got, want = sim.fetch(), oracle_state(o)
        for f in ("x", "y", "z"):
            assert_close(got[f], want[f], 1e-6, 0.0, atol=1e-6, what=f)
        for f in ("v_x", "v_y", "v_z"):
            assert_close(got[f], want[f], 1e-5, 2e-5, what=f)
        assert_close(got["density"], want["density"], 1e-5, 0.0, what="density")
        assert sim.device_errors() == 0
