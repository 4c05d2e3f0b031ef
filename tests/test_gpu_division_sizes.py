"""Division on the device where its work distribution changes: one mother, a few (less than
a warp, one more than a block), and more mothers and daughters than the kernels have blocks
(148 x 8), against the oracle bit for bit (the draws and distances use correctly rounded
operations only, on both sides)."""
import numpy as np
import pytest

from test_gpu_parity import DIV_KW, dividing_state, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_long", [(2, 1), (64, 31), (400, 129), (1300, 1300)])
def test_division_of_few_and_of_all_cells(n, n_long):
    cells, _ = dividing_state(n=n, seed=50 + n, n_long=n_long, crowd=n > 100)
    sim, o = make_pair(cells, cap_cells=2 * n, **DIV_KW)
    parents = -np.ones(n, dtype=np.int32)
    sim.set_parents(parents)
    o.set_parents(parents)
    sim.set_clock(0.25, 1e-6, 17)
    nd = sim.divide_cells()
    tries = o.divide(0.25, 17)
    assert nd == n_long and sim.num_cells() == n + n_long
    assert sim.last_division_tries() == tries
    assert np.array_equal(sim.download_cells(), o.cells())
    assert np.array_equal(sim.parents(), o.parents())
    sim.close()
