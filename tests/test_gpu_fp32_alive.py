"""The FP32 pair kernel on species with alive flags, and the currents of species
of one ragged chunk, against the scalar FP32 form (the persistent ensemble
kernel steps the same species): one and two pairs per lane, whole dead groups of
64 particles (a warp with nothing to step), dead beside live ones in a pair, and
both in the last lane.

Tolerance: test_gpu_fp32_pairs.py's.  Positions within 1e-5 cell, velocities
within 1e-5 c, J within 1e-5 of max|J| (ten roundings of each deposit in another
order).  Dead particles and the flags: bit for bit.
"""
import numpy as np
import pytest

from helpers import rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W
from test_gpu_fp64_lanes import mixed_species

pytestmark = pytest.mark.gpu

SLOTS = 148 * 16 * 32  # lanes resident on a B200
KEYS = ("r", "z", "vr", "vphi", "vz")


def flags(n, seed):
    rng = np.random.default_rng(seed)
    alive = (rng.uniform(size=n) < 0.7).astype(np.uint8)
    alive[128:320] = 0  # three groups of 64, one and a half chunks of 128
    alive[-2:] = (1, 0) if n % 2 == 0 else (0, 1)
    return alive


@pytest.mark.parametrize("with_flags", [False, True])
@pytest.mark.parametrize("n,pusher", [(3, "boris"), (127, "vay"), (130, "boris_classic"),
                                      (8 * SLOTS - 1, "boris"), (8 * SLOTS + 131, "boris"),
                                      (8 * SLOTS + 130, "vay"), (8 * SLOTS + 2, "boris_classic")])
def test_pairs_against_the_scalar_form(n, pusher, with_flags):
    wl = W.small_config(pusher=pusher)
    sp = mixed_species(wl, n, seed=n % 1000)
    if pusher == "boris_classic":  # u = gamma v / c is its speed: below c
        sp.vr, sp.vphi, sp.vz = 0.4 * sp.vr, 0.4 * sp.vphi, 0.4 * sp.vz
    wl.species = [sp]
    pair, scalar = [api.from_workload(wl, precision="fp32") for _ in range(2)]
    alive = flags(n, n) if with_flags else np.ones(n, dtype=np.uint8)
    before = pair.species(0)
    for s in (pair, scalar):
        seed_fields([s], (wl.n_grid_r, wl.n_grid_z), seed=3)
        if with_flags:
            s.set_species(0, alive=alive)
    pair.step()
    pair.sync()
    ens = api.Ensemble([scalar])
    ens.run(1)
    a, b = pair.species(0), scalar.species(0)
    assert np.array_equal(a["alive"], alive) and np.array_equal(b["alive"], alive)
    for k, tol in zip(KEYS, (1e-5 * wl.dr, 1e-5 * wl.dz) + (1e-5 * W.LIGHT_SPEED,) * 3):
        assert np.array_equal(a[k][alive == 0], before[k][alive == 0]), k
        assert np.abs(a[k] - b[k]).max() <= tol, k
    for c in ("J_r", "J_phi", "J_z"):
        assert scalar.field(c).any()
        assert rel_inf(pair.field(c), scalar.field(c)) <= 1e-5, c
    ens.close()
    pair.close()
    scalar.close()
