"""The FP64 particle kernel and the charge weighting at the ends of the number
range: speeds whose square overflows, positions whose cell number does, a
particle that passes exactly through the axis.  What the CPU step refuses or
steps, they refuse or step.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

V_GE_C, OUT_OF_GRID = 4, 5


def one_particle(wl, **kw):
    """A particle at rest amid the grid, but for the values in kw."""
    s = {"r": 5.3 * wl.dr, "z": 7.4 * wl.dz, "vr": 0.0, "vphi": 0.0, "vz": 0.0, "w": 1e4, **kw}
    return W.SpeciesInit("Electrons", -1.0, 1.0, *[np.atleast_1d(np.asarray(s[k], dtype=float))
                                                   for k in ("r", "z", "vr", "vphi", "vz", "w")])


@pytest.mark.parametrize("pusher", ["boris", "vay"])
@pytest.mark.parametrize("component,speed", [("vr", 1e160), ("vphi", -1e200), ("vz", 1.7e308),
                                             ("vz", 3.1e8)])
def test_speeds_above_c_are_refused(component, speed, pusher):
    wl = W.small_config(pusher=pusher)
    wl.species = [one_particle(wl, **{component: speed})]
    sim = api.from_workload(wl)
    sim.step()
    assert sim.status() == V_GE_C
    sim.close()


@pytest.mark.parametrize("axis", ["r", "z"])
@pytest.mark.parametrize("x", [1.0, 1e200, 1e306, 1.7e308])
def test_positions_far_outside_are_refused(axis, x):
    wl = W.small_config()
    wl.species = [one_particle(wl, **{axis: x})]
    sim = api.from_workload(wl)
    sim.step()
    assert sim.status() == OUT_OF_GRID
    sim.close()


@pytest.mark.parametrize("axis", ["r", "z"])
@pytest.mark.parametrize("x", [1.0, 1e306, 1.7e308])
def test_charge_of_far_positions_is_refused(axis, x):
    wl = W.small_config()
    wl.species = [one_particle(wl, **{axis: x})]
    sim = api.from_workload(wl)
    sim.charge_density()
    assert sim.status() == OUT_OF_GRID
    sim.close()


@pytest.mark.parametrize("pusher", ["boris", "vay", "boris_classic"])
def test_a_particle_on_the_axis(pusher):
    """Starts on the axis: at the mid-step its radius is 0, its current is not a
    number there, and its own step ends where the CPU step ends it."""
    wl = W.small_config(pusher=pusher)
    wl.species = [one_particle(wl, r=np.zeros(2), z=np.array([5.3, 12.6]) * wl.dz,
                               vr=np.zeros(2), vphi=np.zeros(2), vz=np.array([0.0, 2e7]),
                               w=np.full(2, 1e4))]
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    orc.step()
    gpu.step()
    a, b = gpu.species(0), orc.species(0)
    assert np.isfinite(b["r"]).all()
    for k in ("r", "z", "vr", "vphi", "vz"):
        assert np.array_equal(a[k], b[k]), k
    for c in GRIDS:
        assert np.array_equal(np.isnan(gpu.field(c)), np.isnan(orc.field(c))), c
    gpu.close()
