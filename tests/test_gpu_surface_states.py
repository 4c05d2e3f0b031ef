"""Velocities and an RK attempt of cells at the edges of the surface contact's cases: clear of
the surface, touching it to within rounding, the lower end in it, both ends in it, upright,
nearly horizontal and lying on it, with and without Coulomb truncation, against the oracle.
Cells stand alone, so that every force is the surface's.

Bar: 1e-10 normwise per column, the FP64 bar of the other parity tests.  The closed forms of
the contact integrals lose up to 1 / rho^3 digits, rho = h n_z / (R - r_z); the states keep
rho >= 0.02, so rounding stays below 2e-16 / 8e-6 = 3e-11."""
import numpy as np
import pytest

import abm_b200
import oracle_ref as orc
from test_gpu_parity import colwise_relerr

pytestmark = pytest.mark.gpu
R = 0.8
JKR = orc.jkr_table(R, 0.5, 3900.0, 100.0, 100)


def surface_states(seed):
    rng = np.random.default_rng(seed)
    rows = []
    for nz in (1.0, 0.999, 0.6, 0.1, 0.01, 1e-3):
        for h in (0.7, 1.9, 2.8):
            low = h * nz
            for rz in (R + low + 0.5, R + low, R + low - 1e-3, R + low - min(0.05, 1.5 * low),
                       R - 0.02, R - 0.05):
                rows.append((rz, nz, h))
    for h in (0.7, 2.8):
        for rz in (R + 0.1, R - 0.03):
            rows.append((rz, 0.0, h))
    n = len(rows)
    c = np.zeros((n, 22), order="F")
    for k, (rz, nz, h) in enumerate(rows):
        az = rng.uniform(0, 2 * np.pi)
        c[k, 0] = k
        c[k, 1:4] = (20.0 * (k % 12), 20.0 * (k // 12), rz)
        c[k, 4:7] = (np.sqrt(1 - nz * nz) * np.cos(az), np.sqrt(1 - nz * nz) * np.sin(az), nz)
        c[k, 13], c[k, 14] = 2 * h, h
        c[k, 17], c[k, 18], c[k, 19], c[k, 20], c[k, 21] = 100.0, 720.0, 100.0, 1, 100.0
    c[:, 7:13] = rng.normal(0.0, 5.0, (n, 6))
    return c


@pytest.mark.parametrize("coulomb", [0.0, 0.05, 1.0])
@pytest.mark.parametrize("method", [abm_b200.HEUN_EULER, abm_b200.DORMAND_PRINCE])
def test_velocities_at_the_edges_of_contact(coulomb, method):
    cells = surface_states(5)
    sim = abm_b200.Simulation(cap_cells=len(cells), jkr_table=JKR, cell_surface_coulomb_coeff=coulomb,
                              integration_mode=method)
    sim.upload_cells(cells)
    o = orc.Oracle(sim.pdict, jkr=JKR)
    o.set_cells(cells)
    assert sim.get_cell_neighbors() == o.build_neighbors()
    assert colwise_relerr(sim.get_velocities(), o.get_velocities()) <= 1e-10
    assert colwise_relerr(sim.step_runge_kutta_adaptive(1e-8)[0], o.rk_attempt(1e-8)[0]) <= 1e-10
    sim.close()
