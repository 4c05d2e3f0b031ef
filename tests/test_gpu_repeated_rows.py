"""Neighbor rows from the caller that list a pair more than once: every listed row adds its
force, as a walk over the reference's table does, in 3-D and 2-D."""
import numpy as np
import pytest

import abm_b200
import oracle_ref as orc
from abm_b200 import workloads
from test_gpu_parity import RTOL, colwise_relerr, make_pair, patch_state

pytestmark = pytest.mark.gpu


def repeated(rows, seed):
    rng = np.random.default_rng(seed)
    times = rng.choice([1, 1, 1, 2, 5], len(rows))
    out = np.repeat(rows, times, axis=0)
    return out[rng.permutation(len(out))]


def forces_equal(sim, want):
    for _ in range(2):                       # a pass that lists the active pairs, and one over them
        assert colwise_relerr(sim.cell_cell_forces(), want) <= RTOL
    sim.close()


@pytest.mark.parametrize("n", [40, 3000])
def test_repeated_rows_3d(n):
    sim, o = make_pair(patch_state(n, 60 + n))
    o.build_neighbors()
    rows = repeated(o.neighbors(), 4)
    sim.set_neighbors(rows)
    o.set_neighbors(rows)
    forces_equal(sim, o.cell_cell_forces())


def test_every_row_twice_2d():
    cells = workloads.biofilm_2d(500, seed=8)
    params = dict(abm_b200.DEFAULTS_2D, Ldiv=4.4, neighbor_threshold=3.2, adhesion_mode=1, adhesion_strength=20.0,
                  adhesion_mindist=1.2)
    sim = abm_b200.Simulation(cap_cells=500, **params)
    sim.upload_cells(cells)
    o = orc.Oracle2D(sim.pdict)
    o.set_cells(cells)
    o.build_neighbors()
    sim.set_neighbors(np.concatenate([o.neighbors(), o.neighbors()]))
    forces_equal(sim, 2 * o.cell_cell_forces())
