"""The neighbor build and the division as a cooperative grid: launches are shaped for twice the
cells (at most cap_cells), and a shape of more than 8,192 cells is a grid, so these contexts have
that much room.  Pair set, distances and daughters equal the oracle's bit for bit."""
import numpy as np
import pytest

import abm_b200
import oracle_ref as orc
from abm_b200 import workloads
from test_gpu_build_sizes import table_equals
from test_gpu_parity import DIV_KW, dividing_state, make_pair, patch_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 6001, 20011])
def test_grid_build_3d(n):
    table_equals(*make_pair(patch_state(n, 700 + n), cap_cells=2 * n + 16))


def test_grid_build_2d():
    cells = workloads.biofilm_2d(4500, seed=45)
    sim = abm_b200.Simulation(cap_cells=9100, **dict(abm_b200.DEFAULTS_2D, Ldiv=4.4, neighbor_threshold=3.2))
    sim.upload_cells(cells)
    o = orc.Oracle2D(sim.pdict)
    o.set_cells(cells)
    table_equals(sim, o)


@pytest.mark.parametrize("n_long", [1, 700, 5000])
def test_grid_division(n_long):
    cells, _ = dividing_state(n=5000, seed=90 + n_long, n_long=n_long)
    sim, o = make_pair(cells, cap_cells=12000, **DIV_KW)
    parents = -np.ones(5000, dtype=np.int32)
    sim.set_parents(parents)
    o.set_parents(parents)
    sim.set_clock(0.25, 1e-6, 17)
    assert sim.divide_cells() == n_long
    tries = o.divide(0.25, 17)
    assert sim.last_division_tries() == tries
    assert np.array_equal(sim.download_cells(), o.cells())
    assert np.array_equal(sim.parents(), o.parents())
    assert sim.get_cell_neighbors() == o.build_neighbors()
    assert np.array_equal(sim.neighbors(), o.neighbors())
    sim.close()
