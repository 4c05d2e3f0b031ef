"""Large frames and tables come to the host in pieces by several threads: sizes below the
split, at it, and with a ragged last piece; whole ranges and rows of a larger array; a
destination in pinned memory; and several contexts downloading at once."""
import threading

import numpy as np
import pytest

import abm_b200
from test_gpu_parity import patch_state

pytestmark = pytest.mark.gpu


def context(n, seed):
    base = patch_state(1000, seed)
    cells = np.asfortranarray(np.tile(base, (-(-n // 1000), 1))[:n])
    cells[:, 0] = np.arange(n)
    cells[:, 1] += 1e3 * (np.arange(n) // 1000)
    cells[:, 7:13] = np.random.default_rng(seed).normal(size=(n, 6))
    sim = abm_b200.Simulation(cap_cells=n, cap_neighbors_per_cell=64)
    sim.upload_cells(cells)
    return sim, cells


@pytest.mark.parametrize("n", [1000, 71493, 71494, 100003])     # 22 columns: 12 MiB lies at 71,493.8 cells
def test_frames_arrive_whole(n):
    sim, cells = context(n, n)
    assert np.array_equal(sim.download_cells(), cells)
    wide = np.full((n + 77, 22), -1.0, order="F")               # rows of a larger array
    sim.download_cells_raw(wide.ctypes.data, n + 77)
    assert np.array_equal(wide[:n], cells) and (wide[n:] == -1.0).all()
    import torch
    pinned = torch.zeros(22, n, dtype=torch.float64, pin_memory=True)
    sim.download_cells_raw(pinned.data_ptr(), n)
    assert np.array_equal(pinned.numpy().T, cells)
    sim.close()


def test_contexts_download_side_by_side():
    made = [context(80000 + 17 * k, k) for k in range(4)]
    good = [False] * 4

    def look(k):
        good[k] = all(np.array_equal(made[k][0].download_cells(), made[k][1]) for _ in range(3))

    threads = [threading.Thread(target=look, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(good)
    for sim, _ in made:
        sim.close()
