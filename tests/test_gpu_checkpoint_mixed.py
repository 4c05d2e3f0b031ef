"""Exact checkpoints in mixed precision: how a pass rounds its FP32 distances depends on the
motion since the pass before a rebuild, which the file keeps, so a resumed run ends bit for bit
where the uninterrupted one ends; a file without that block still loads."""
import os

import numpy as np
import pytest

import abm_b200
from abm_b200 import stepsize
from test_gpu_checkpoint import DIV_KW, JKR, STATS, growing_state

pytestmark = pytest.mark.gpu


def new_sim(n, controller):
    sim = abm_b200.Simulation(jkr_table=JKR, cap_cells=3 * n, max_stepsize=1e-3, iter_update_neighbors=10,
                              controller=controller, precision=abm_b200.PRECISION_MIXED, **DIV_KW)
    if controller == abm_b200.CONTROLLER_LEARNED:
        sim.set_stepsize_weights(stepsize.load())
    return sim


def begun(cells, controller):
    sim = new_sim(len(cells), controller)
    sim.upload_cells(cells)
    sim.set_parents(-np.ones(len(cells), dtype=np.int32))
    sim.set_clock(0.0, 1e-4, 0)
    sim.get_cell_neighbors()
    return sim


# 17: between two rebuilds; 20: just after one
@pytest.mark.parametrize("at", [17, 20])
@pytest.mark.parametrize("controller", [abm_b200.CONTROLLER_REFERENCE, abm_b200.CONTROLLER_LEARNED,
                                        abm_b200.CONTROLLER_PI])
def test_mixed_run_resumes_bit_for_bit(controller, at, tmp_path):
    cells = growing_state(400, 35)
    a = begun(cells, controller)
    sa = a.iterate(35)
    b = begun(cells, controller)
    b.iterate(at)
    path = os.fspath(tmp_path / "run.ckpt")
    b.save_checkpoint(path)
    c = new_sim(400, controller)
    c.load_checkpoint(path)
    sc = c.iterate(35 - at)
    assert a.clock() == c.clock()
    assert np.array_equal(a.parents(), c.parents())
    assert np.array_equal(a.download_cells(), c.download_cells())
    for k in STATS:
        assert sa[k] == sc[k], k
    for sim in (a, b, c):
        sim.close()


def test_file_without_the_mixed_block(tmp_path):
    cells = growing_state(300, 36)
    b = begun(cells, abm_b200.CONTROLLER_REFERENCE)
    b.iterate(7)
    path = os.fspath(tmp_path / "run.ckpt")
    b.save_checkpoint(path)
    blob = bytearray(open(path, "rb").read())
    head = np.frombuffer(bytes(blob[8:32]), dtype=np.int32).copy()
    assert head[5] == 1
    n, ncols, m, parents = b.num_cells(), b.ncols, head[3], head[4]
    tail = 8 * n * ncols + 8 * m + 4 * parents            # cells, pairs, lineage
    head[5] = 0
    plain = bytes(blob[:8]) + head.tobytes() + bytes(blob[32:len(blob) - tail - 16]) + bytes(blob[len(blob) - tail:])
    with open(path, "wb") as f:
        f.write(plain)
    c = new_sim(300, abm_b200.CONTROLLER_REFERENCE)
    c.load_checkpoint(path)
    assert np.array_equal(b.download_cells(), c.download_cells()) and b.clock() == c.clock()
    assert c.iterate(5)["iterations"] == 12
    head[5] = 2
    with open(path, "wb") as f:
        f.write(bytes(blob[:8]) + head.tobytes() + bytes(blob[32:]))
    with pytest.raises(RuntimeError, match="ABM_ERR_ARG"):
        c.load_checkpoint(path)
    b.close()
    c.close()
