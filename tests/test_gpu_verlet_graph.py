"""Velocity-Verlet steps in graphs of ten, alone and unlaunched by graphs: the same kernels on the
same data, so the states must agree bit for bit, for counts below, at and beyond ten steps,
with divisions and a periodic rebuild among them and with a stop at a cell count."""
import numpy as np
import pytest

import abm_b200
from abm_b200 import workloads

pytestmark = pytest.mark.gpu


def run(calls, stop=0, **kw):
    n = 300
    cells, _ = workloads.biofilm_3d(n=n, seed=6, disk_radius=300.0 * np.sqrt(n / 1e5) + 4.0, lmax=5.6, p_contact=0.9)
    cells[:, 16] = 1.5
    cells[::25, 13] = 5.6 - 1e-4 * np.arange(1, 13)
    cells[::25, 14] = cells[::25, 13] / 2
    sim = abm_b200.Simulation(cap_cells=4 * n, integration_mode=abm_b200.VELOCITY_VERLET, M0=30.0, L0=2.0,
                              max_stepsize=1e-5, growth_mean=1.5, growth_std=0.1, daughter_length_std=0.01,
                              daughter_angle_xy_bound=0.05, daughter_angle_z_bound=0.05, rng_seed=3,
                              iter_update_neighbors=20, **kw)
    sim.upload_cells(cells)
    sim.set_parents(-np.ones(n, dtype=np.int32))
    sim.set_clock(0.0, 1e-5, 0)
    for k in calls:
        sim.iterate(k, stop)
    out = sim.download_cells(), sim.parents(), sim.stats()
    info = sim.graph_info()
    sim.close()
    return out, info


@pytest.mark.parametrize("count", [9, 10, 11, 43])
def test_verlet_graphs_match_single_steps(count):
    one, info = run([count])
    assert info == "conditional"
    assert count < 43 or one[2]["divisions"] > 0
    for other in (run([1] * count)[0], run([count], use_graphs=0)[0]):
        assert np.array_equal(one[0], other[0]) and np.array_equal(one[1], other[1])
        assert one[2] == other[2]


def test_verlet_stop_at_a_cell_count_is_the_same_step():
    one, plain = run([60], stop=301)[0], run([60], stop=301, use_graphs=0)[0]
    assert one[2]["n_cells"] >= 301 and one[2]["iterations"] < 60
    assert np.array_equal(one[0], plain[0]) and one[2] == plain[2]
