"""Calls recorded into a graph and run again without the library seeing it: the
cell data of a recorded neighbour search are those of the present slots, and stage
functions, recorded or called after a replay, give the states of plain calls bit
for bit."""
import numpy as np
import pytest

from sphpc_b200 import Simulation

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "x_star", "y_star", "z_star", "v_x", "v_y", "v_z", "dp_x", "dp_y", "dp_z",
          "w_x", "w_y", "w_z", "color_x", "color_y", "color_z", "density", "lambda")
SOLVE = (("compute_densities",), ("compute_lambda",), ("update_dps", 0), ("update_position_stars",))
POST = (("update_velocities",), ("surface_tension",), ("apply_viscosity",), ("compute_vorticity",),
        ("vorticity_confinement",))


def call(sim, ops):
    for op, *args in ops:
        getattr(sim, op)(*args)


def record(sim, ops):
    """The calls as a graph on the set's stream, and that stream."""
    import torch
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        call(sim, ops)
    return graph, stream


def replay(graph, stream, times):
    import torch
    with torch.cuda.stream(stream):
        for _ in range(times):
            graph.replay()


def test_cell_data_after_a_replay():
    with Simulation("small_dam") as sim:
        sim.step(20)
        sim.find_all_neighbors()
        want = sim.cell_data()
        # an even number of searches leaves the state in the buffers it was in
        graph, stream = record(sim, (("find_all_neighbors",),) * 2)
        for _ in range(3):
            replay(graph, stream, 1)
            for got, w in zip(sim.cell_data(), want):
                np.testing.assert_array_equal(got, w)
        assert np.all(np.diff(want[0].astype(np.int64)) >= 0)
        assert sim.device_errors() == 0
        graph.reset()


def started(sim):
    sim.step(3)
    call(sim, (("apply_gravity",), ("predict_positions",), ("find_all_neighbors",)))


def test_recorded_stages_equal_plain_calls():
    with Simulation("small_dam") as a, Simulation("small_dam") as b:
        started(a)
        call(a, SOLVE * 7 + POST)
        started(b)
        graph, stream = record(b, SOLVE * 2)
        replay(graph, stream, 1)
        call(b, SOLVE * 2)      # plain calls between two replays and after them
        replay(graph, stream, 1)
        call(b, SOLVE + POST)
        got, want = b.fetch(), a.fetch()
        for f in FIELDS:
            np.testing.assert_array_equal(np.asarray(got[f]), np.asarray(want[f]), err_msg=f)
        graph.reset()
