"""The loop graph (rounds of plain iterations, a full one only where divisions, the cell limit
or a failed first attempt ask for it) against single-iteration graphs and against launches
without graphs: the same kernels on the same data, so the states must agree bit for bit, for
iteration counts below, at and beyond the length of a round.  The start step is far too long,
so the first iterations retry; cells at the division length divide along the way."""
import numpy as np
import pytest

import abm_b200
from abm_b200 import stepsize, workloads

pytestmark = pytest.mark.gpu


def run(calls, controller, limit=0, **kw):
    n = 500
    cells, _ = workloads.biofilm_3d(n=n, seed=9, disk_radius=300.0 * np.sqrt(n / 1e5) + 4.0, lmax=5.6, p_contact=0.9)
    cells[:, 16] = 1.5
    # a step adds some 1e-5 um: these reach the division length after a few to some tens of steps
    cells[::50, 13] = 5.6 - 3e-5 * np.arange(1, 11)
    cells[::50, 14] = cells[::50, 13] / 2
    sim = abm_b200.Simulation(cap_cells=4 * n, controller=controller, max_stepsize=1e-4, growth_mean=1.5,
                              growth_std=0.1, daughter_length_std=0.01, daughter_angle_xy_bound=0.05,
                              daughter_angle_z_bound=0.05, rng_seed=3, **kw)
    if controller == abm_b200.CONTROLLER_LEARNED:
        sim.set_stepsize_weights(stepsize.load())
    sim.upload_cells(cells)
    sim.set_parents(-np.ones(n, dtype=np.int32))
    sim.set_clock(0.0, 1e-4, 0)
    if limit:
        sim.set_cell_limit(limit)
    for k in calls:
        sim.iterate(k)
    out = sim.download_cells(), sim.parents(), sim.stats()
    sim.close()
    return out


@pytest.mark.parametrize("controller", [0, 1, 2])
@pytest.mark.parametrize("count", [4, 8, 9, 43])
def test_loop_graph_matches_single_iterations(controller, count):
    one = run([count], controller)
    many = run([1] * count, controller)
    plain = run([count], controller, use_graphs=0)
    assert one[2]["retries"] + one[2]["rejected"] > 0
    assert count < 43 or one[2]["divisions"] > 0
    for other in (many, plain):
        assert np.array_equal(one[0], other[0]) and np.array_equal(one[1], other[1])
        assert one[2] == other[2]


def test_loop_graph_stops_at_the_cell_limit():
    free = run([60], 0)
    assert free[2]["n_cells"] > 501
    one = run([60], 0, limit=501)
    many = run([1] * 60, 0, limit=501)
    assert one[2]["n_cells"] >= 501 and one[2]["iterations"] < 60
    assert np.array_equal(one[0], many[0]) and one[2] == many[2]
