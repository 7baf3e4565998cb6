"""Stage functions called in unusual orders: the records that one stage leaves
for the next never change a result.  Each sequence runs twice, once with a query
between all calls (after which every stage makes its own records); the states are
equal bit for bit."""
import numpy as np
import pytest

from sphpc_b200 import Simulation

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "x_star", "y_star", "z_star", "v_x", "v_y", "v_z", "dp_x", "dp_y", "dp_z",
          "w_x", "w_y", "w_z", "color_x", "color_y", "color_z", "density", "lambda")
SOLVE = ("compute_densities", "compute_lambda", "update_dps", "update_position_stars")


def run(sequence, query):
    with Simulation("small_dam") as sim:
        sim.step(3)
        sim.apply_gravity()
        sim.predict_positions()
        sim.find_all_neighbors()
        for op in SOLVE:
            getattr(sim, op)(*((0,) if op == "update_dps" else ()))
        for op in sequence:
            if query:
                assert sim.device_errors() == 0
            if op.startswith("push "):
                f = op.split()[1]
                sim.push({f: sim.fetch()[f] * 1.25})
            else:
                getattr(sim, op)(*((1,) if op == "update_dps" else ()))
        return sim.fetch()


@pytest.mark.parametrize("sequence", [
    SOLVE * 2,
    ("compute_lambda", "compute_densities", "update_dps", "update_dps", "update_position_stars"),
    ("compute_vorticity", "update_dps", "compute_densities", "vorticity_confinement"),
    ("compute_densities", "surface_tension", "compute_densities", "apply_viscosity",
     "compute_vorticity", "surface_tension", "vorticity_confinement", "compute_lambda"),
    ("compute_lambda", "push lambda", "update_dps", "update_position_stars", "compute_densities"),
    ("surface_tension", "push density", "apply_viscosity", "compute_lambda", "update_dps"),
    ("update_velocities", "apply_viscosity", "update_positions", "apply_viscosity",
     "predict_positions", "compute_densities", "compute_lambda"),
    ("predict_positions", "compute_densities", "find_all_neighbors", "compute_lambda",
     "step", "compute_densities", "compute_lambda", "update_dps"),
], ids=lambda s: "+".join(w.split()[-1][:8] for w in s))
def test_records_between_stages_change_nothing(sequence):
    a, b = run(sequence, False), run(sequence, True)
    for f in FIELDS:
        np.testing.assert_array_equal(np.asarray(a[f]), np.asarray(b[f]), err_msg=f)
