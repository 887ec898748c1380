"""pdp3g_get_species on both sides of its size rule: small states packed into
one copy (sizes that end inside an 8-byte word of the alive array), larger ones
array by array into pages already present and into fresh ones.  Whole values:
what was set comes back bit for bit.
"""
import numpy as np
import pytest

from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 9, 5340, 5400, 300001])  # 49 bytes each: the line is at 5349
def test_species_come_back_as_set(n):
    wl = W.small_config()
    rng = np.random.default_rng(n)
    r, z = rng.uniform(wl.dr, wl.r_size - wl.dr, n), rng.uniform(wl.dz, wl.z_size - wl.dz, n)
    v, w = rng.normal(0.0, 1e6, (3, n)), rng.uniform(1e3, 1e4, n)
    wl.species = [W.SpeciesInit("Electrons", -1.0, 1.0, r, z, *v, w)]
    sim = api.from_workload(wl)
    alive = (rng.uniform(size=n) < 0.7).astype(np.uint8)
    sim.set_species(0, alive=alive)
    for _ in range(2):
        got = sim.species(0)
        want = {"r": r, "z": z, "vr": v[0], "vphi": v[1], "vz": v[2], "w": w, "alive": alive}
        for k, a in want.items():
            assert np.array_equal(got[k], a), k
    sim.close()
