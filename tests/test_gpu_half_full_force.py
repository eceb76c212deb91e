"""A full-list force over half lists whose build is still in flight, followed by the final and the next
initial integration (the calls that run fused in a full-list step): positions, velocities and forces are
the oracle's bit for bit, whether or not the lists were read in between."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu


def state(lib, product, cells, half_mode, read):
    set_mode = lib.md_set_half_mode if hasattr(lib, "md_set_half_mode") else lib.oracle_set_half_mode
    set_mode(half_mode)
    try:
        sim = make_sim(lib, cells=cells, setup_lib=product)
        sim.step(0.005, 3)  # the last list build whose status was read is a full one
        lib.md_assemble_neighborlists(True, sim.cell)
        if read:
            tinymd.neighbor_lists(lib, sim.n, 512)
        lib.md_compute_lennard_jones(False, sim.cutoff, sim.eps, sim.sigma)
        lib.md_final_integration(0.005)
        lib.md_initial_integration(0.005)
        lib.md_synchronize_ghost_layer()
        got = tinymd.full_state(lib)
        sim.close()
    finally:
        set_mode(0)
    return got


# 16, 8, 4 lanes per atom and one, with the next gathers in flight
@pytest.mark.parametrize("half_mode", [0, 1])
@pytest.mark.parametrize("cells", [(4, 4, 4), (9, 10, 8), (14, 15, 16), (22, 22, 22)])
def test_full_force_fused_over_half_lists(product, oracle, cuda_device, cells, half_mode):
    expected = state(oracle, product, cells, half_mode, False)
    for read in (False, True):
        for a, b in zip(state(product, product, cells, half_mode, read), expected):
            np.testing.assert_array_equal(a, b)
