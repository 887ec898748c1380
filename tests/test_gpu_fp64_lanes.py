"""The FP64 particle kernel against the oracle where its own rules switch: the
particles per lane (1, 2 or 4 by the species' size) with ragged last warps, and
the general deposition path beside the in-cell one (steps that cross faces,
radial moves of more than a 32nd of the radius, starts exactly on cell faces
and half cells, where the gather and the deposition change branch).

Tolerance: the FP64 form's one-step bound, every grid within 1e-12 of max|x|
and every particle array within 1e-12.  Positions are the oracle's bit for bit
but for particles whose velocity differs by an ulp (gather weights): at most a
few of a species, each moving J by 1e-11 of its own share, which is below 1e-4
of max|J| for the populations here.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload, rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

SLOTS = 148 * 8 * 64  # lanes resident on a B200


def mixed_species(wl, n, seed):
    """n electrons: a third thermal, a third fast (up to 0.9 c), a third
    starting exactly on radial or axial faces and half cells."""
    rng = np.random.default_rng(seed)
    dr, dz = wl.dr, wl.dz
    r = rng.uniform(dr / 2, wl.r_size - dr / 2, n)
    z = rng.uniform(dz / 2, wl.z_size - dz / 2, n)
    kind = np.arange(n) % 3
    lat = kind == 2
    r[lat] = (rng.integers(2, 2 * wl.n_grid_r - 4, lat.sum()) * 0.5) * dr
    z[lat] = (rng.integers(2, 2 * wl.n_grid_z - 4, lat.sum()) * 0.5) * dz
    v = rng.normal(0.0, 4e5, (3, n))
    d = rng.normal(size=(3, n))
    d *= rng.uniform(0.05, 0.9, n) * W.LIGHT_SPEED / np.sqrt((d * d).sum(0))
    v = np.where(kind == 1, d, v)
    return W.SpeciesInit("Electrons", -1.0, 1.0, r, z, *v, rng.uniform(0.5e4, 2e4, n))


@pytest.mark.parametrize("n,pusher", [(1, "boris"), (33, "vay"), (2 * SLOTS - 1, "boris"),
                                      (2 * SLOTS + 1, "vay"), (8 * SLOTS + 129, "boris"),
                                      (8 * SLOTS + 2, "boris_classic")])
def test_one_step_equals_the_oracle(n, pusher):
    wl = W.small_config(pusher=pusher)
    wl.species = [mixed_species(wl, n, seed=n % 1000)]
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    seed_fields([orc, gpu], (wl.n_grid_r, wl.n_grid_z), seed=3)
    orc.step()
    gpu.step()
    gpu.sync()
    for c in GRIDS:
        assert rel_inf(gpu.field(c), orc.field(c)) <= 1e-12, c
    a, b = gpu.species(0), orc.species(0)
    for k in ("r", "z", "vr", "vphi", "vz"):
        assert float(np.abs(a[k] - b[k]).max()) <= 1e-12 * float(np.abs(b[k]).max()), k
