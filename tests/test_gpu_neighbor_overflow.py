"""More neighbors than a row holds: the build reports it and leaves an empty neighbor set, so
that nothing later walks rows whose entries lack their partners, also inside a running loop."""
import ctypes

import numpy as np
import pytest

import abm_b200
from test_gpu_parity import DIV_KW, JKR, patch_state

pytestmark = pytest.mark.gpu


def pairs_after_overflow(sim):
    s = abm_b200.AbmStats()
    rc = abm_b200.LIB.abm_get_stats(sim._ctx, ctypes.byref(s))
    assert abm_b200.ERRORS[rc] == "ABM_ERR_CAPACITY"
    return s.n_pairs


def largest_row(cells):
    sim = abm_b200.Simulation(jkr_table=JKR, cap_cells=len(cells))
    sim.upload_cells(cells)
    sim.get_cell_neighbors()
    most = np.bincount(sim.neighbors()[:, :2].astype(int).ravel()).max()
    sim.close()
    return int(most)


# one cluster, and a cooperative grid (launches are shaped for twice the cells); one row too
# long, and nearly all of them
@pytest.mark.parametrize("n", [300, 5000])
@pytest.mark.parametrize("short_by", [1, None])
def test_overflow_leaves_no_table(n, short_by):
    cells = patch_state(n, 900 + n)
    rows = largest_row(cells) - short_by if short_by else 3
    sim = abm_b200.Simulation(jkr_table=JKR, cap_cells=n if n < 1000 else 2 * n, cap_neighbors_per_cell=rows)
    sim.upload_cells(cells)
    with pytest.raises(RuntimeError, match="ABM_ERR_CAPACITY.*cap_neighbors_per_cell"):
        sim.get_cell_neighbors()
    assert pairs_after_overflow(sim) == 0
    for call in (sim.cell_cell_forces, sim.neighbors):
        with pytest.raises(RuntimeError, match="ABM_ERR_STATE"):
            call()
    sim.close()


# eight parallel cells side by side, 1.3 um apart: at most four neighbors within 3.6 um; once
# all have divided, an inner daughter has four beside it and five of the other halves
@pytest.mark.parametrize("graphs", [1, 0])
def test_overflow_inside_the_loop(graphs):
    cells = np.zeros((8, 22), order="F")
    cells[:, 0] = np.arange(8)
    cells[:, 2], cells[:, 3] = 1.3 * np.arange(8), 5.0
    cells[:, 4] = 1.0
    cells[:, 13], cells[:, 14] = 5.6 + 1e-3, 2.8 + 5e-4
    cells[:, 16:22] = 1.5, 100.0, 720.0, 100.0, 1.0, 100.0
    assert largest_row(cells) == 4
    sim = abm_b200.Simulation(jkr_table=JKR, cap_cells=64, cap_neighbors_per_cell=4, use_graphs=graphs, **DIV_KW)
    sim.upload_cells(cells)
    sim.set_parents(-np.ones(8, dtype=np.int32))
    assert sim.get_cell_neighbors() == 13
    with pytest.raises(RuntimeError, match="ABM_ERR_CAPACITY.*cap_neighbors_per_cell"):
        sim.iterate(12)
    assert pairs_after_overflow(sim) == 0
    sim.close()
