"""Batches of colonies whose launches are cooperative grids: each context's grids take its share
of the chip, so that the contexts run side by side; the shape changes no result."""
import time

import numpy as np
import pytest

import abm_b200
from abm_b200 import replicates, workloads

pytestmark = pytest.mark.gpu


def context(n, seed, growing, **kw):
    p = dict(replicates.CONFIG0, cap_cells=2 * n + 64, rng_seed=seed, max_stepsize=1e-4 if growing else 1e-6, **kw)
    if not growing:
        p.update(growth_mean=0.0, growth_std=0.0)
    cells = workloads.biofilm_2d(n, seed=seed, lmin=1.4, lmax=4.4 if growing else 4.3)
    cells[:, 12] = 1.5 if growing else 0.0
    sim = abm_b200.Simulation(**p)
    sim.upload_cells(cells)
    sim.set_parents(-np.ones(n, dtype=np.int32))
    sim.set_clock(0.0, 1e-6, 0)
    sim.get_cell_neighbors()
    return sim


# launches are shaped for twice the cells: all three are grids, the last with a tile of its own;
# 23 iterations: two rounds of the loop graph and a few single iterations
def test_batch_of_grids_matches_contexts_advanced_alone():
    kw = [dict(), dict(iter_update_neighbors=100), dict(pair_tile=512, pair_blocks_per_sm=2)]
    sizes = [4500, 6001, 5200]
    alone = [context(n, n, True, **k) for n, k in zip(sizes, kw)]
    batched = [context(n, n, True, **k) for n, k in zip(sizes, kw)]
    batch = abm_b200.Batch(batched)
    for calls in (20, 3):
        batch.iterate(calls)
    batch.synchronize()
    for a, b in zip(alone, batched):
        a.iterate(23)
        assert a.stats() == b.stats() and a.stats()["divisions"] > 0
        assert np.array_equal(a.download_cells(), b.download_cells())
        assert np.array_equal(a.neighbors(), b.neighbors())
    # a context is on its own again outside the batch
    batched[1].iterate(5)
    alone[1].iterate(5)
    assert np.array_equal(alone[1].download_cells(), batched[1].download_cells())
    batch.close()
    for s in alone + batched:
        s.close()


def us_per_iteration(advance, wait, iters=100):
    best = 1e9
    for _ in range(4):
        t = time.perf_counter()
        advance(iters)
        wait()
        best = min(best, (time.perf_counter() - t) * 1e6 / iters)
    return best


# eight colonies of 20,000 cells at rest: 56 us an iteration, 108 with grids of the whole chip,
# against 26 of one colony alone
def test_batch_of_grids_runs_side_by_side():
    sims = [context(20000, 30 + k, False) for k in range(8)]
    one = us_per_iteration(lambda k: sims[0].iterate(k, stats=False), sims[0].synchronize)
    batch = abm_b200.Batch(sims)
    eight = us_per_iteration(batch.iterate, batch.synchronize)
    batch.close()
    for s in sims:
        s.close()
    print("one colony %.1f us, eight %.1f us" % (one, eight))
    assert eight < 3.5 * one
