"""A colony that has reached its cell limit takes no further step, but the calls that evaluate
its present state (forces, velocities, one attempt) answer for that state, also after its
neighbors have been built again."""
import numpy as np
import pytest

import abm_b200
import oracle_ref as orc
from test_gpu_friction import monolayer, pair, with_friction
from test_gpu_parity import RTOL, colwise_relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rebuild", [False, True])
def test_calls_at_the_cell_limit(rebuild):
    cells = with_friction(monolayer(n_side=16), 0, 73)
    cells[:, 7:13] = 0.0
    cells[:, 7:9] = np.random.default_rng(3).normal(0.0, 0.5, (len(cells), 2))
    sim, o = pair(cells, adhesion_mode=0, max_rz_noise=3000.0, rng_seed=11, growth_mean=1.0)
    assert sim.get_cell_neighbors() == o.build_neighbors()
    sim.set_cell_limit(len(cells))
    assert sim.iterate(3)["iterations"] == 0
    if rebuild:
        sim.get_cell_neighbors()
    assert colwise_relerr(sim.cell_cell_forces(), o.cell_cell_forces()) <= RTOL
    assert colwise_relerr(sim.get_velocities(), o.get_velocities()) <= RTOL
    got, _, _ = sim.step_runge_kutta_adaptive(2e-4)      # its stages change planar decisions
    want, _, _ = o.rk_attempt(2e-4)
    assert colwise_relerr(got, want) <= RTOL
    assert sim.iterate(3)["iterations"] == 0             # and it still stands
    sim.set_cell_limit(0)
    assert sim.iterate(3)["iterations"] == 3
    sim.close()
