"""The Poisson sweep on both sides of its batches of sixteen rows (one batch, one
and a row, two and a row).

Tolerance: the solve's own, 1e-11 of each grid's largest magnitude.
"""
import numpy as np
import pytest

from oracle.poisson import poisson_dirichlet
from pdp3_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [4, 16, 17, 18, 19, 32, 33, 34, 35])
def test_poisson_matches_the_oracle(nr):
    nz, dr, dz = 15, 4e-4, 5e-4
    rho = np.random.default_rng(nr).normal(0.0, 1e-4, (nr, nz))
    sim = api.Simulation(dr * (nr - 1), dz * (nz - 1), nr, nz, 1e-13)
    phi = sim.poisson_solve(rho)
    for got, ref in zip((phi, sim.field("E_r"), sim.field("E_z")), poisson_dirichlet(rho, dr, dz)):
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    sim.close()
