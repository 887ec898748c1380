"""pdp3g_forward_window advances the context as pdp3g_step does, with other
roundings: the window steps its particles one by one, pdp3g_step two at a time.

Tolerance: a step rounds a particle's offset and momentum by a few 6e-8.  These
particles move by a fiftieth of a cell and more, so that a step's current changes
by at most 4 x 6e-8 x 50 = 1.2e-5 of itself; the fields hold twelve steps of it,
their own part (the seeds) not at all: 1.5e-4 of max|E|, max|H|, and twice that
for the loss, a square.  Positions: 12 x 4 x 6e-8 = 3e-6 cells, doubled by the
velocities', 1e-5.
"""
import numpy as np
import pytest

from helpers import rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 12
PROBE = (2, 12, 6, 24)


def context(beam):
    wl = W.small_config(beam=beam)
    n = 4000
    rng = np.random.default_rng(12)
    r = rng.uniform(wl.dr, wl.r_size - 2 * wl.dr, n)
    z = rng.uniform(wl.dz, wl.z_size - 2 * wl.dz, n)
    d = rng.normal(size=(3, n))
    d *= rng.uniform(0.1, 0.8, n) * W.LIGHT_SPEED / np.sqrt((d * d).sum(0))
    wl.species = [W.SpeciesInit("Electrons", -1.0, 1.0, r, z, *d, rng.uniform(0.5e4, 2e4, n))]
    sim = api.from_workload(wl, precision="fp32")
    seed_fields([sim], (wl.n_grid_r, wl.n_grid_z), seed=9)
    return wl, sim


@pytest.mark.parametrize("interval", [STEPS, 5])
@pytest.mark.parametrize("beam", [False, True])
def test_window_and_steps_end_alike(beam, interval):
    wl, sim = context(beam)
    _, ref = context(beam)
    adj = api.Adjoint(sim, STEPS, interval, PROBE)
    loss = adj.forward()
    ref.step(STEPS)
    ref.sync()
    assert sim.time == ref.time
    for c in ("E_r", "E_phi", "E_z", "H_r", "H_phi", "H_z"):
        assert rel_inf(sim.field(c), ref.field(c)) <= 1.5e-4, c
    assert loss == pytest.approx(W.probe_loss(ref.field("E_z"), wl.dr, wl.dz, PROBE), rel=3e-4)
    for sid in range(2 if beam else 1):
        a, b = sim.species(sid), ref.species(sid)
        assert np.array_equal(a["alive"], b["alive"])
        live = b["alive"] == 1
        for k, cell in (("r", wl.dr), ("z", wl.dz)):
            assert np.abs(a[k] - b[k])[live].max() <= 1e-5 * cell, (sid, k)
    adj.close()
