"""The field kernels over the whole range of a double: the leading tail of a
pulse falls through the smallest normal numbers to zero, an unstable run grows
to infinity.  Fields alone, so every value is the CPU step's bit for bit, the
sign of a zero included; where that is not a number, ours is not.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

SEEDED = ("E_r", "E_phi", "E_z", "H_r", "H_phi", "H_z")


def spread(rng, shape, lo, hi):
    """Magnitudes spread over the exponents lo..hi, either sign, some zeros."""
    a = rng.uniform(1.0, 10.0, shape) * 10.0 ** rng.integers(lo, hi, shape)
    a[rng.uniform(size=shape) < 0.1] = 0.0
    return a * rng.choice([-1.0, 1.0], shape)


def check(fields, steps=3):
    wl = W.small_config(n_grid_r=18, n_grid_z=41)
    wl.species = []
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    for c, a in fields((wl.n_grid_r, wl.n_grid_z)).items():
        orc.set_field(c, a)
        gpu.set_field(c, a)
    orc.run(steps)
    gpu.step(steps)
    gpu.sync()
    for c in GRIDS:
        a, b = gpu.field(c), orc.field(c)
        nan = np.isnan(b)
        assert np.array_equal(np.isnan(a), nan), c
        assert np.array_equal(a[~nan].view(np.uint64), b[~nan].view(np.uint64)), c
    gpu.close()


@pytest.mark.parametrize("lo,hi", [(-322, -270), (-320, 5), (-5, 5), (250, 300)])
def test_magnitudes(lo, hi):
    rng = np.random.default_rng(lo + 1000)
    check(lambda shape: {c: spread(rng, shape, lo, hi) for c in SEEDED})


@pytest.mark.parametrize("component", SEEDED)
def test_infinities(component):
    rng = np.random.default_rng(3)

    def fields(shape):
        out = {c: rng.normal(0.0, 1e3, shape) for c in SEEDED}
        out[component][3, 7], out[component][9, 30], out[component][0, 20] = np.inf, -np.inf, np.inf
        return out

    check(fields, steps=1)
