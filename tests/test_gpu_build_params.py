"""Parameters under which no pair can pass the centre-distance test: the grid still has bins."""
import pytest

from test_gpu_parity import make_pair, patch_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ldiv", [-5.2, -500.0])     # the test's limit: 3.6 + Ldiv + 1.6 um
def test_no_pair_within_the_centre_distance(Ldiv):
    sim, o = make_pair(patch_state(500, 12), Ldiv=Ldiv)
    assert sim.get_cell_neighbors() == o.build_neighbors() == 0
    assert not sim.cell_cell_forces().any()
    sim.close()
