"""The reverse of the particle phase sums a warp's field adjoints by cell: one
cell in the warp, two, or more have each their own path.  The same particles
in another order must give the same gradient.

Tolerance: 1e-4 of each gradient's largest value.  Another order changes the
FP32 partial sums of J (1e-6 of E) and those of the runs (32 x 6e-8), while the
particles' part of the E_r, E_z and H_phi gradients is some hundredths ((omega_p
dt)^2 = 0.05) and that of E_phi, H_r and H_z all of it, so that a sum put on a
wrong node is off by 1e-2 or more.
"""
import numpy as np
import pytest

from helpers import seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

N = 999  # the last warp is not full


def particles(wl):
    """33 cells of particles in cell order, every quadrant of a cell, cells on
    the axis among them."""
    rng = np.random.default_rng(7)
    per = -(-N // 33)
    c = np.repeat(np.arange(33), per)[:N]
    i, k = c % 11, 5 + c // 11
    r = np.maximum((i + rng.uniform(0.02, 0.98, N)) * wl.dr, 0.6 * wl.dr)
    z = (k + rng.uniform(0.02, 0.98, N)) * wl.dz
    d = rng.normal(size=(3, N))
    v = d / np.sqrt((d * d).sum(0)) * rng.uniform(0.05, 0.5, N) * W.LIGHT_SPEED
    return np.vstack([r, z, v])


def gradient(wl, state, weight):
    wl.species = [W.SpeciesInit("Electrons", -1.0, 1.0, *state, np.full(state.shape[1], weight))]
    sim = api.from_workload(wl, precision="fp32")
    seed_fields([sim], (wl.n_grid_r, wl.n_grid_z), seed=4)
    adj = api.Adjoint(sim, 2, 2, (0, 12, 4, 12))
    adj.forward()
    adj.backward()
    out = {c: adj.field(c) for c in ("E_r", "E_phi", "E_z", "H_r", "H_phi", "H_z")}
    adj.close()
    sim.close()
    return out


@pytest.mark.parametrize("order", ["two cells", "four cells", "mixed"])
def test_order_of_the_particles_does_not_matter(order):
    wl = W.small_config()
    state = particles(wl)
    if order == "mixed":
        perm = np.random.default_rng(8).permutation(N)
    else:  # interleave halves or quarters: particles of 2 or 4 cells alternate
        parts = np.array_split(np.arange(N), 2 if order == "two cells" else 4)
        perm = np.array([p[j] for j in range(len(parts[0])) for p in parts if j < len(p)])
    assert np.array_equal(np.sort(perm), np.arange(N))
    want, got = gradient(wl, state, 1e10), gradient(wl, state[:, perm], 1e10)
    for c in want:
        assert np.abs(want[c]).max() > 0, c
        assert np.abs(got[c] - want[c]).max() <= 1e-4 * np.abs(want[c]).max(), c
