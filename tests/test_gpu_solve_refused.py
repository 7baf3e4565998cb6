"""The solve of a small set in one launch with an obstacle, against the passes
launched one by one: positions, velocities and density are equal bit for bit.  The
passes run where the cooperative launch is refused (injected on the host: the error
that the driver gives on a stream with a part of the device), which is no error of
the step, and in the adaptive driver with a tolerance that is never met."""
import numpy as np
import pytest

from sphpc_b200 import Simulation, _lib

pytestmark = pytest.mark.gpu
ITERATIONS = {"small_dam": 4, "small_obstacle": 6}
FIELDS = ("x", "y", "z", "v_x", "v_y", "v_z", "density")


def run(name, refuse=0, steps=3, **solver):
    """State, steps of the solve in one launch, passes over the positions."""
    lib = _lib.load()
    with Simulation(name, solver_overrides=solver) as sim:
        rng = np.random.default_rng(11)
        sim.push({f: 4.0 * rng.uniform(-1, 1, sim.n) for f in ("v_x", "v_y", "v_z")})
        sim.profile(True)
        try:
            assert lib.sphpc_fail_solve_launch(refuse) == 0
            sim.step(steps)
        finally:
            lib.sphpc_fail_solve_launch(0)
        times = sim.profile_read()
        assert sim.device_errors() == 0
        state = sim.fetch()
        return {f: np.asarray(state[f]) for f in FIELDS}, times.get("position", (0,))[0]


@pytest.mark.parametrize("name", ["small_dam", "small_obstacle"])
@pytest.mark.parametrize("solver", [dict(), dict(scorr_k=0.0), dict(scorr_n=3)])
def test_refused_launch_takes_the_passes(name, solver):
    want, passes = run(name, **solver)
    assert passes == 0
    for refuse, expected in ((3, 3), (1, 1)):
        got, passes = run(name, refuse, **solver)
        assert passes == ITERATIONS[name] * expected
        for f in FIELDS:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)


@pytest.mark.parametrize("name", ["small_dam", "small_obstacle"])
def test_one_launch_equals_the_adaptive_passes(name):
    """Positions and density; the adaptive driver forms its velocities from the
    rounded displacement, the solve from the exact one: one rounding apart."""
    want, _ = run(name, steps=1)
    got, passes = run(name, steps=1, adaptive=1, density_tolerance=-1.0,
                      max_iterations=ITERATIONS[name], min_progress=0.0)
    assert passes == ITERATIONS[name]
    for f in ("x", "y", "z", "density"):
        np.testing.assert_array_equal(got[f], want[f], err_msg=f)


def test_injection_rejects_bad_arguments():
    assert _lib.load().sphpc_fail_solve_launch(-1) != 0
    assert _lib.load().sphpc_fail_solve_launch(0) == 0
