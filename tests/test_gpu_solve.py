"""The solve of a small set in one launch against the same passes launched one by
one (the adaptive driver with a tolerance that is never met runs those): positions
and density after a step are equal bit for bit, for the pressure terms and an
obstacle, at the set sizes where the launch changes."""
import numpy as np
import pytest

from sphpc_b200 import Simulation
from sphpc_b200.scenes import config_path

pytestmark = pytest.mark.gpu


def scene(tmp_path, dims, **solver):
    text = open(config_path("small_dam")).read()
    text = text.replace("number_particles = 4096", f"number_particles = {dims[0] * dims[1] * dims[2]}")
    for axis, m, old_box in zip("xyz", dims, (48.0, 24.0, 24.0)):
        text = text.replace(f"max_{axis} = {old_box}", f"max_{axis} = {1.5 * m + 4:.9g}")
        text = text.replace(f"max_{axis} = 16.0", f"max_{axis} = {float(m):.9g}")
    path = tmp_path / "scene.ini"
    path.write_text(text)
    return Simulation(str(path), solver_overrides=solver)


@pytest.mark.parametrize("dims,scorr_k,scorr_n,iterations", [
    ((3, 3, 3), 0.001, 4, 4),           # one block, not full
    ((4, 8, 4), 0.001, 4, 1),           # one block, full
    ((43, 3, 1), 0.0, 4, 3),            # two blocks; without the pressure term
    ((16, 16, 16), 0.001, 3, 16),       # the most iterations of one launch
    ((16, 16, 16), 0.001, 4, 17),       # one more: pass by pass
    ((31, 33, 37), 0.001, 4, 4),        # an odd count
    ((37, 64, 32), 0.001, 4, 3),        # 75,776: four blocks an SM
    ((47, 41, 41), 0.001, 4, 3),        # more
])
def test_solve_in_one_launch_equals_its_passes(tmp_path, dims, scorr_k, scorr_n, iterations):
    common = dict(scorr_k=scorr_k, scorr_n=scorr_n)
    with scene(tmp_path, dims, solve_iterations=iterations, **common) as a, \
            scene(tmp_path, dims, adaptive=1, density_tolerance=-1.0, max_iterations=iterations,
                  min_progress=0.0, **common) as b:
        rng = np.random.default_rng(5)
        jolt = {f: 3.0 * rng.uniform(-1, 1, a.n) for f in ("v_x", "v_y", "v_z")}
        for sim in (a, b):
            sim.push(jolt)
            sim.step(1)
        got, want = a.fetch(), b.fetch()
        for f in ("x", "y", "z", "density"):
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
        assert a.last_step_info()["iterations"] == b.last_step_info()["iterations"] == iterations
        assert a.device_errors() == 0
