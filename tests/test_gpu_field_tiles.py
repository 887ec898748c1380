"""The field kernels at the edges of their 32 x 8 tiles, and the per-cell
deposits' way into J at every border of the grid.

* Fields only: three graph-replayed steps equal the oracle's bit for bit (the
  divisions are correctly rounded ones).
* The FP32 form's J after one step from seeded fields within 1e-5 of max|J| of
  the scalar FP32 form's (the persistent ensemble kernel, whose deposits go
  straight into J; ten roundings of each deposit in another order), at every
  node: the particles fill the domain up to all four walls.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload, rel_inf, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3), (8, 32), (9, 33), (7, 31), (16, 64), (17, 65)]


def workload(nr, nz, ppc):
    wl = W.small_config(n_grid_r=nr, n_grid_z=nz, r_size=6.25e-4 * (nr - 1),
                        z_size=1.25e-3 * (nz - 1), ppc=ppc)
    wl.pml = None if min(nr, nz) < 8 else wl.pml
    return wl


@pytest.mark.parametrize("nr,nz", SHAPES)
def test_fields_alone(nr, nz):
    wl = workload(nr, nz, 1)
    wl.species = []
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    seed_fields([orc, gpu], (nr, nz), seed=11)
    orc.run(3)
    gpu.step(3)
    gpu.sync()
    for c in GRIDS:
        assert np.array_equal(gpu.field(c), orc.field(c)), c
    assert gpu.time == orc.time


@pytest.mark.parametrize("nr,nz", SHAPES[1:])
def test_fp32_currents_to_the_borders(nr, nz):
    wl = workload(nr, nz, 16)
    gpu, run = (api.from_workload(wl, precision="fp32") for _ in range(2))
    seed_fields([gpu, run], (nr, nz), seed=5)
    gpu.step()
    gpu.sync()
    ens = api.Ensemble([run])
    ens.run(1)
    for c in ("J_r", "J_phi", "J_z"):
        assert np.abs(run.field(c)).max() > 0
        assert rel_inf(gpu.field(c), run.field(c)) <= 1e-5, c
    ens.close()
