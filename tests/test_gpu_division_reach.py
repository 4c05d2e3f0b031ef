"""Division beside a cell so long that the rings of bins around a mother would exceed any grid:
the search covers the whole grid, and the daughters equal the oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import DIV_KW, dividing_state, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1e4, 1e12])
def test_division_beside_a_very_long_cell(half):
    cells, idx = dividing_state(n=400, seed=23, n_long=60)
    k = next(i for i in range(400) if i not in idx)
    cells[k, 1:7] = 0.0, 0.0, 50.0, 1.0, 0.0, 0.0
    cells[k, 14] = half
    sim, o = make_pair(cells, cap_cells=800, **DIV_KW)
    parents = -np.ones(400, dtype=np.int32)
    sim.set_parents(parents)
    o.set_parents(parents)
    sim.set_clock(0.25, 1e-6, 17)
    assert sim.divide_cells() == 60
    tries = o.divide(0.25, 17)
    assert sim.last_division_tries() == tries
    assert np.array_equal(sim.download_cells(), o.cells())
    sim.close()
