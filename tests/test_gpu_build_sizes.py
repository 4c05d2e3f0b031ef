"""The neighbor build where its shape changes: one block, a cluster of blocks, the largest
cluster and the first cooperative grid (launches are shaped for twice the cells), boxes that
need coarse bins, boxes far from the origin, cells of very uneven length, cells in a line and
in a heap, in 3-D and 2-D.  The pair set and the distances must equal the oracle's bit for
bit; the search only drops pairs that its bounds prove too far apart."""
import numpy as np
import pytest

import abm_b200
import oracle_ref as orc
from abm_b200 import workloads
from test_gpu_parity import make_pair, patch_state

pytestmark = pytest.mark.gpu


def table_equals(sim, o):
    m = sim.get_cell_neighbors()
    assert m == o.build_neighbors()
    assert np.array_equal(sim.neighbors(), o.neighbors())
    sim.close()
    return m


@pytest.mark.parametrize("n", [3, 31, 257, 2049, 4096, 4097, 6001])
def test_build_sizes_3d(n):
    table_equals(*make_pair(patch_state(n, 700 + n)))


def shaped(kind):
    cells = patch_state(1500, 77)
    rng = np.random.default_rng(5)
    if kind == "far":                       # FP32 positions lose digits only relative to the box
        cells[:, 1:4] += (3e6, -7e6, 2e5)
    elif kind == "line":                    # more bins of the usual size than the bin capacity
        cells[:, 1] = np.arange(len(cells)) * 700.0 + rng.uniform(0, 2, len(cells))
        cells[1::2, 1] = cells[0::2, 1] + rng.uniform(0.5, 6.0, len(cells) // 2)
        cells[:, 2:4] = rng.uniform(0, 3, (len(cells), 2))
    elif kind == "corners":                 # two clumps 1e6 um apart on every axis
        cells[::2, 1:4] += 1e6
    elif kind == "heap":                    # everything within a few bins
        cells = cells[:150]
        cells[:, 1:4] = rng.uniform(0, 9, (len(cells), 3))
    elif kind == "lengths":                 # a few cells far longer than the others
        cells[::50, 13] = 40.0
        cells[::50, 14] = 20.0
    return cells


@pytest.mark.parametrize("kind", ["far", "line", "corners", "heap", "lengths"])
def test_build_boxes(kind):
    assert table_equals(*make_pair(shaped(kind))) > 0


@pytest.mark.parametrize("n", [1, 40, 4097])
def test_build_sizes_2d(n):
    cells = workloads.biofilm_2d(n, seed=n)
    params = dict(abm_b200.DEFAULTS_2D, Ldiv=4.4, neighbor_threshold=3.2)
    sim = abm_b200.Simulation(cap_cells=n, **params)
    sim.upload_cells(cells)
    o = orc.Oracle2D(sim.pdict)
    o.set_cells(cells)
    table_equals(sim, o)
