"""Alive flags given to a species that had none, after the work that keeps the
species' arrays has been set up: the captured step, the ensemble's descriptors
and its own step graph, the adjoint's stored states.

A dead particle is not pushed: its state stays what it was, bit for bit, while
the others move.  The captured step is also held against the phases launched one
by one, and (FP64) against the oracle.

Tolerance of the grids: the FP64 form's after a few steps, 1e-10 of max|x|; the
FP32 form's deposits are summed in another order by the two paths, which moves
the fields by 1e-16 and a float offset by its last bit (6e-8 of a cell) now and
then, below 1e-4 of max|J| here.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload, rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

KEYS = ("r", "z", "vr", "vphi", "vz")


def dead_third(n):
    alive = np.ones(n, dtype=np.uint8)
    alive[::3] = 0
    return alive


def kill(sim, sid=0):
    """Flags a third of species sid dead; the flags and the dead ones' state."""
    before = sim.species(sid)
    alive = dead_third(before["r"].size)
    sim.set_species(sid, alive=alive)
    return alive, {k: before[k][alive == 0] for k in KEYS}


def check_dead(sim, alive, state, sid=0):
    now = sim.species(sid)
    assert np.array_equal(now["alive"], alive)
    for k in KEYS:
        assert np.array_equal(now[k][alive == 0], state[k]), k
    return now


def fresh(precision, **kw):
    wl = W.small_config(**kw)
    sim = api.from_workload(wl, precision=precision)
    seed_fields([sim], (wl.n_grid_r, wl.n_grid_z), seed=2)
    return wl, sim


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_step_after_flags(precision):
    wl, sim = fresh(precision)
    _, eager = fresh(precision)
    eager.set_timing(True)  # phase by phase, never captured
    for s in (sim, eager):
        s.step(2)
        alive, state = kill(s)
        s.step(3)
        s.sync()
        check_dead(s, alive, state)
    tol = 1e-10 if precision == "fp64" else 1e-4
    for c in GRIDS:
        assert rel_inf(sim.field(c), eager.field(c)) <= tol, c
    if precision == "fp64":
        orc = oracle_from_workload(wl)
        seed_fields([orc], (wl.n_grid_r, wl.n_grid_z), seed=2)
        orc.run(2)
        orc.set_species(0, alive=alive)
        orc.run(3)
        for c in GRIDS:
            assert rel_inf(sim.field(c), orc.field(c)) <= tol, c
    sim.close()
    eager.close()


@pytest.mark.parametrize("mode", ["persistent", "step_graph"])
def test_ensemble_after_flags(mode):
    sims = [fresh("fp32", seed=s)[1] for s in (7, 8)]
    ens = api.Ensemble(sims)
    ens.set_mode(mode)
    ens.run(2)
    alive, state = kill(sims[1])
    other = sims[0].species(0)
    ens.run(3)
    now = check_dead(sims[1], alive, state)
    assert np.any(now["r"][alive == 1] != other["r"][alive == 1])
    assert np.any(sims[0].species(0)["r"] != other["r"])
    ens.close()


def test_adjoint_after_flags():
    _, sim = fresh("fp32")
    _, ref = fresh("fp32")
    adj = api.Adjoint(sim, 4, 2, (2, 10, 6, 20))
    adj.forward()
    ref_adj = api.Adjoint(ref, 4, 2, (2, 10, 6, 20))
    ref_adj.forward()
    alive, state = kill(sim)
    kill(ref)
    ref_adj.close()  # this one is made again, for a species that has flags
    ref_adj = api.Adjoint(ref, 4, 2, (2, 10, 6, 20))
    loss, want = adj.forward(), ref_adj.forward()
    assert loss == pytest.approx(want, rel=1e-4)
    adj.backward()
    check_dead(sim, alive, state)
    g = adj.species(0)
    for k in ("r", "z", "ur", "uphi", "uz"):
        assert not g[k][alive == 0].any(), k
        assert g[k][alive == 1].any(), k
    ref_adj.close()
    adj.close()


def test_adjoint_refuses_other_species():
    wl, sim = fresh("fp32")
    adj = api.Adjoint(sim, 4, 2, (2, 10, 6, 20))
    adj.forward()
    s = wl.species[0]
    sim.add_species(s.charge_e, s.mass_me, s.r, s.z, s.vr, s.vphi, s.vz, s.w)
    for call in (adj.forward, adj.backward):
        with pytest.raises(api.Pdp3gError) as e:
            call()
        assert e.value.status == 1
    adj.close()


@pytest.mark.parametrize("mode", ["persistent", "step_graph"])
def test_ensemble_steps_a_species_added_later(mode):
    wl, sim = fresh("fp32")
    ens = api.Ensemble([sim])
    ens.set_mode(mode)
    ens.run(1)
    s = wl.species[0]
    sid = sim.add_species(s.charge_e, s.mass_me, s.r, s.z, s.vr, s.vphi, s.vz, s.w)
    before = sim.species(sid)
    ens.run(2)
    assert np.any(sim.species(sid)["r"] != before["r"])
    assert ens.info()["particles"] == sum(sim.species_size(j) for j in range(sid + 1))
    ens.close()
