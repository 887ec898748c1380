"""A diagnostics call that finds device memory for a part of its scratch only:
it reports that, and so does the next one; with memory again the same context
gives its results.
"""
import numpy as np
import pytest

from pdp3_b200 import api

pytestmark = pytest.mark.gpu

NO_MEMORY = 8


def test_scratch_that_fits_in_part():
    torch = pytest.importorskip("torch")
    small = api.Simulation(1e-2, 4e-2, 17, 33, 1e-13)
    small.charge_density()  # the kernels are loaded before memory is short
    small.diagnostics()
    nr, nz = 2049, 4097
    grid = 8 * nr * nz  # 64 MiB: one more fits, the second does not
    sim = api.Simulation(1.0, 2.0, nr, nz, 1e-13)
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - grid * 3 // 2, dtype=torch.uint8, device="cuda")
    try:
        free, _ = torch.cuda.mem_get_info()
        assert grid < free < 2 * grid
        for call in (sim.charge_density, sim.charge_density, sim.diagnostics):
            with pytest.raises(api.Pdp3gError) as e:
                call()
            assert e.value.status == NO_MEMORY
    finally:
        del hold
        torch.cuda.empty_cache()
    assert not sim.charge_density().any()
    sim.set_field("E_z", np.ones((nr, nz)))
    assert sim.diagnostics()["field_energy"] > 0
    small.close()
    sim.close()
