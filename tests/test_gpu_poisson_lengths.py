"""The Poisson solve at every kind of transform length: 8 (one trip of three
stages), 16 and 32 (a trip of one and of two stages left), 256, 4096 and 8192
(two groups per thread), and grids of few rows and of rows that are no multiple
of the sweep's eight.

Tolerance: the solve's own, 1e-11 of each grid's largest magnitude.
"""
import numpy as np
import pytest

from oracle.poisson import poisson_dirichlet
from pdp3_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz", [(3, 3), (9, 7), (10, 15), (33, 127), (40, 2047), (18, 4095)])
def test_poisson_matches_the_oracle(nr, nz):
    dr, dz = 4e-4, 5e-4
    rng = np.random.default_rng(nz)
    rho = rng.normal(0.0, 1e-4, (nr, nz))
    sim = api.Simulation(dr * (nr - 1), dz * (nz - 1), nr, nz, 1e-13)
    phi = sim.poisson_solve(rho)
    want = poisson_dirichlet(rho, dr, dz)
    for got, ref in zip((phi, sim.field("E_r"), sim.field("E_z")), want):
        assert np.abs(ref).max() > 0
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    sim.close()
