"""Device blocks kept between grids: grids of changing sizes, each on blocks that an earlier and
larger or smaller grid left behind, stay bit-identical to the CPU oracle; md_mpi_finalize gives the
kept blocks back to the device."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [False, True])
def test_grids_of_changing_sizes_on_kept_blocks(product, oracle, cuda_device, half):
    for cells in ((8, 8, 8), (4, 4, 4), (9, 7, 5), (8, 8, 8)):
        got = []
        for lib in (product, oracle):
            sim = make_sim(lib, cells=cells, half=half, setup_lib=product)
            sim.step(0.005, 21)
            got.append(tinymd.full_state(lib))
            sim.close()
        for a, b in zip(*got):
            if half:  # atomics: the summation order is free (the half lists' tolerance of test_gpu_parity.py)
                np.testing.assert_allclose(a, b, rtol=0, atol=1e-10 * max(1.0, np.abs(b).max()))
            else:
                np.testing.assert_array_equal(a, b)


def test_finalize_gives_the_kept_blocks_back(product, cuda_device):
    import torch

    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info(cuda_device)[0]

    product.md_mpi_finalize()  # whatever earlier grids left
    before = free_bytes()
    sim = make_sim(product, cells=(32, 32, 32), setup_lib=product)
    held = product.md_device_bytes()
    sim.close()
    kept = before - free_bytes()
    assert kept <= (1 << 30) + (64 << 20)  # bounded (plus the driver's granularity)
    product.md_mpi_finalize()
    left = before - free_bytes()
    assert left < held // 4  # what stays is the driver's own, not the grid's blocks
    # and the library goes on afterwards
    sim = make_sim(product, cells=(4, 4, 4), setup_lib=product)
    sim.step(0.005, 3)
    sim.close()
    tinymd.check(product)
