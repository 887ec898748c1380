"""The kinetic energy of one particle, to the last bit: m c^2 beta^2 / (s (1 + s)),
s = sqrt(1 - beta^2), and in the cell-local form m c^2 u^2 / (sqrt(1 + u^2) + 1),
each operation correctly rounded.  One velocity component with an exact square,
so that the sum of squares holds no rounding of its own.
"""
import numpy as np
import pytest

from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

C2 = 9.0e16


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_single_particles(precision):
    wl = W.small_config()
    w = 12345.0
    wl.species = [W.SpeciesInit("Electrons", -1.0, 1.0, *[np.array([x]) for x in (
        3.3 * wl.dr, 9.2 * wl.dz, 0.0, 0.0, 0.0, w)])]
    sim = api.from_workload(wl, precision=precision)
    mass = 1.0 * 9.1e-31
    rng = np.random.default_rng(17)
    wrong = []
    for v in 4.0 * rng.integers(1000, 7 * 10 ** 7, 300):
        assert v * v == float(int(v) ** 2) and v < 3e8
        sim.set_species(0, vr=np.array([v]))
        if precision == "fp64":
            b2 = v * v / C2
            s = np.sqrt(1.0 - b2)
            want = mass * w * C2 * b2 / (s * (1.0 + s))
        else:
            u = float(np.float32(v * (1.0 / (3.0e8 * np.sqrt(1.0 - v * v / C2)))))
            want = mass * w * C2 * (u * u) / (np.sqrt(1.0 + u * u) + 1.0)
        got = sim.diagnostics()["kinetic_energy"]
        if got != want:
            wrong.append((v, got, want))
    assert not wrong, (len(wrong), wrong[:3])
    sim.close()
