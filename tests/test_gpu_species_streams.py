"""The particle phase with one to seven species: on one, two and three streams
and with several species on a stream, sizes in and out of order, with a bunch,
as a captured step and phase by phase, and in the form for species of 2^20
particles and more.

Tolerance: the FP64 form's after a few steps, every grid within 1e-10 of
max|x| of the oracle's (one step: 1e-12, growing with the fields they feed).
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload, rel_inf
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu


def some_species(wl, sizes):
    out = []
    for j, n in enumerate(sizes):
        rng = np.random.default_rng(j)
        r = rng.uniform(wl.dr, wl.r_size - 2 * wl.dr, n)
        z = rng.uniform(wl.dz, wl.z_size - 2 * wl.dz, n)
        v = rng.normal(0.0, 2e6, (3, n))
        out.append(W.SpeciesInit("Electrons", -1.0 if j % 2 == 0 else 1.0, 1.0 + 3 * j, r, z, *v,
                                 rng.uniform(0.5e4, 2e4, n)))
    return out


@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("sizes,beam", [((300,), False), ((500, 20), False), ((400, 900), True),
                                        ((64, 2000, 7, 300), True), ((5, 4, 3, 2, 1, 6), True),
                                        (((1 << 20) + 3, 100), True)])
def test_steps_equal_the_oracle(sizes, beam, timing):
    wl = W.small_config(beam=beam, steps=3)
    wl.species = some_species(wl, sizes)
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    gpu.set_timing(timing)
    for _ in range(3):
        orc.step()
    gpu.step(3)
    gpu.sync()
    for c in GRIDS:
        assert rel_inf(gpu.field(c), orc.field(c)) <= 1e-10, c
    gpu.close()
