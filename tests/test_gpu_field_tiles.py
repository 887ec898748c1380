"""The field kernels at the edges of their 32 x 8 tiles: three graph-replayed
steps of the fields alone equal the oracle's bit for bit (the divisions are
correctly rounded ones).  The per-cell deposits' way into J, up to the borders
of the grid, is checked in test_gpu_fp32_pairs.py.
"""
import numpy as np
import pytest

from helpers import GRIDS, oracle_from_workload, seed_fields
from pdp3_b200 import api
from pdp3_b200 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3), (8, 32), (9, 33), (7, 31), (16, 64), (17, 65)]


@pytest.mark.parametrize("nr,nz", SHAPES)
def test_fields_alone(nr, nz):
    wl = W.small_config(n_grid_r=nr, n_grid_z=nz, r_size=6.25e-4 * (nr - 1),
                        z_size=1.25e-3 * (nz - 1), ppc=1)
    wl.pml = None if min(nr, nz) < 8 else wl.pml
    wl.species = []
    orc, gpu = oracle_from_workload(wl), api.from_workload(wl)
    seed_fields([orc, gpu], (nr, nz), seed=11)
    orc.run(3)
    gpu.step(3)
    gpu.sync()
    for c in GRIDS:
        assert np.array_equal(gpu.field(c), orc.field(c)), c
    assert gpu.time == orc.time
