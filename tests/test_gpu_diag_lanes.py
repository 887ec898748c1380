"""The charge, density, temperature and kinetic-energy passes where their lanes
change rule: species that end inside a lane's four particles or a warp's 128,
one that needs a second round of CTAs, runs of one cell and of changing cells,
particles on faces, half cells and next to the axis.

Tolerance: the node sums have positive terms (charge and density: 1e-12 of the
largest value, as the density's own test); the temperature within 1e-12 of its
largest value plus the rounding bound of the order of its sums; the energy is a
sum of at most 6.1e5 positive terms of a few roundings each (1e-9 covers the
order's worst case, 6.1e5 x 1.1e-16).
"""
import numpy as np
import pytest

from oracle.diagnostics import particles_density, temperature_classic
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

ROUND = 148 * 4 * 256 * 4  # particles of one round of CTAs on a B200


def species(wl, n, seed):
    rng = np.random.default_rng(seed)
    dr, dz = wl.dr, wl.dz
    r = rng.uniform(0.01 * dr, wl.r_size - dr, n)
    z = rng.uniform(0.01 * dz, wl.z_size - dz, n)
    near = np.arange(n) % 7 == 3
    r[near] = rng.uniform(0.01, 1.2, near.sum()) * dr
    lat = np.arange(n) % 5 == 2
    r[lat] = rng.integers(1, 2 * wl.n_grid_r - 4, lat.sum()) * 0.5 * dr
    z[lat] = rng.integers(1, 2 * wl.n_grid_z - 4, lat.sum()) * 0.5 * dz
    run = (np.arange(n) // 50) % 2 == 1  # every other fifty share a cell
    r[run], z[run] = 3.3 * dr, 4.6 * dz
    v = rng.normal(0.0, 2e6, (3, n))
    return W.SpeciesInit("Electrons", -1.0, 1.0, r, z, *v, rng.uniform(0.5e4, 2e4, n))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [1, 3, 127, 128, 130, ROUND + 1022])
def test_grids_and_energy(n, precision):
    wl = W.small_config()
    wl.species = [species(wl, n, seed=n % 1000)]
    sim = api.from_workload(wl, precision=precision)
    sp, m, q = sim.species(0), 9.1e-31, 1.6e-19
    args = (wl.dr, wl.dz, wl.n_grid_r, wl.n_grid_z)
    want = particles_density(sp["r"], sp["z"], m * sp["w"], *args)
    top = np.abs(want).max()
    assert np.abs(sim.density(0) - want).max() <= 1e-12 * top
    assert np.abs(sim.charge_density(1) + q * want).max() <= 1e-12 * q * top
    ref, rnd = temperature_classic(sp["r"], sp["z"], sp["vr"], sp["vphi"], sp["vz"], *args, m, q,
                                   rounding=True)
    got, fin = sim.temperature(0)[:-1, :-1], ~np.isnan(ref)
    assert np.array_equal(np.isnan(got), ~fin)
    assert np.all(np.abs(got - ref)[fin] <= 1e-12 * np.abs(ref[fin]).max() + rnd[fin])
    d = sim.diagnostics()
    b2 = (sp["vr"] ** 2 + sp["vphi"] ** 2 + sp["vz"] ** 2) / W.LIGHT_SPEED ** 2
    root = np.sqrt(1 - b2)
    kin = float((m * W.LIGHT_SPEED ** 2 * sp["w"] * b2 / (root * (1 + root))).sum())
    assert abs(d["kinetic_energy"] - kin) <= 1e-9 * kin
    assert d["alive"] == n
    sim.close()
