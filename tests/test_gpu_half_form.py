"""The form that half lists are built in depends on the grid's own force, not on what an earlier grid of
the process ran: a grid issues the same kernels whether an LJ or a DEM grid was there before it."""
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu

FORCES = {"lj": dict(cells=(7, 8, 9)),
          "dem": dict(benchmark="granular_gas", cells=(9, 8, 9), cutoff=1.2, force_field="dem",
                      dem=(0.1, 0.1, 100.0, 0.5))}


def launches(lib, force):
    """Kernels of a grid's first lists and force, and of turning those lists into the reference's for a read"""
    lib.md_set_dem_model(1 if force == "dem" else 0, 0.6)
    try:
        sim = make_sim(lib, half=True, setup_lib=lib, **FORCES[force])
        lib.md_synchronize()
        first = lib.md_kernel_launches()
        tinymd.neighbor_lists(lib, sim.n, 512)
        read = lib.md_kernel_launches() - first
        sim.close()
    finally:
        lib.md_set_dem_model(0, 1.0)
    return first, read


@pytest.mark.parametrize("force", ["lj", "dem"])
def test_form_of_the_first_half_lists(product, cuda_device, force):
    seen = {}
    for before in ("lj", "dem"):
        launches(product, before)
        seen[before] = launches(product, force)
    assert seen["lj"] == seen["dem"]
