"""The FP32 pair kernel where its rules switch: one or two pairs per lane (by
the species' size) with ragged last chunks, particles that leave the packed
in-cell path (cell crossings, walls, large radial moves) beside ones that stay
in it, unsorted cells inside a lane, and a species of more than one chunk per
resident warp.

* A particle's own step does not depend on its place: the first 4097 particles
  of a large species end, bit for bit, where they end as a species of their own
  (which takes one pair per lane).
* Against the FP64 oracle: positions within 1e-5 cell and momenta within 1e-5
  of the largest speed (a hundred FP32 roundings of offsets in (0, 1]).
* J against the scalar FP32 form (the persistent ensemble kernel steps the same
  species): within 1e-5 of max|J|, ten roundings of each deposit in another
  order.  Not against the oracle: the upstream deposits nothing for a step that
  passes exactly through a cell corner (src/particles.cpp:560-680 tests z1 < z2
  and z1 > z2 only), as some of these starts do, and the cell-local form does.
"""
import numpy as np
import pytest

from helpers import oracle_from_workload, rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W
from test_gpu_fp64_lanes import mixed_species

pytestmark = pytest.mark.gpu

SLOTS = 148 * 16 * 32  # lanes resident on a B200
KEYS = ("r", "z", "vr", "vphi", "vz")


def step(wl, species):
    wl.species = [species]
    gpu = api.from_workload(wl, precision="fp32")
    seed_fields([gpu], (wl.n_grid_r, wl.n_grid_z), seed=3)
    gpu.step()
    gpu.sync()
    return gpu


@pytest.mark.parametrize("n,pusher", [(3, "boris"), (127, "vay"), (8 * SLOTS - 1, "boris"),
                                      (8 * SLOTS + 1, "vay"), (8 * SLOTS + 131, "boris")])
def test_pairs_against_the_oracle_and_alone(n, pusher):
    wl = W.small_config(pusher=pusher)
    sp = mixed_species(wl, n, seed=n % 1000)
    gpu = step(wl, sp)
    orc = oracle_from_workload(wl)
    seed_fields([orc], (wl.n_grid_r, wl.n_grid_z), seed=3)
    orc.step()
    a, b = gpu.species(0), orc.species(0)
    # starts on a face round to either side of it in FP32: compared in cells
    assert np.abs(a["r"] - b["r"]).max() <= 1e-5 * wl.dr
    assert np.abs(a["z"] - b["z"]).max() <= 1e-5 * wl.dz
    for k in ("vr", "vphi", "vz"):
        assert np.abs(a[k] - b[k]).max() <= 1e-5 * W.LIGHT_SPEED, k
    if n > 1000:
        run = api.from_workload(wl, precision="fp32")
        seed_fields([run], (wl.n_grid_r, wl.n_grid_z), seed=3)
        ens = api.Ensemble([run])
        ens.run(1)
        for c in ("J_r", "J_phi", "J_z"):
            assert rel_inf(gpu.field(c), run.field(c)) <= 1e-5, c
        ens.close()
        m = 4097
        few = W.SpeciesInit(sp.name, sp.charge_e, sp.mass_me,
                            *[getattr(sp, k)[:m] for k in KEYS + ("w",)])
        alone = step(wl, few).species(0)
        for k in KEYS:
            assert np.array_equal(a[k][:m], alone[k]), k
