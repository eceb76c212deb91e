"""Device memory that a closed grid leaves with the library goes back to the device when the program asks
for it, without ending the library or touching an open grid."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu


def free_bytes(device):
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(device)[0]


def test_blocks_of_a_closed_grid_are_released(product, cuda_device):
    tinymd.release_device_memory(product)
    before = free_bytes(cuda_device)
    sim = make_sim(product, cells=(32, 32, 32), setup_lib=product)
    held = product.md_device_bytes()
    sim.close()
    tinymd.release_device_memory(product)
    assert before - free_bytes(cuda_device) < held // 4  # what stays is the driver's own
    tinymd.check(product)


def test_an_open_grid_is_not_touched(product, oracle, cuda_device):
    make_sim(product, cells=(16, 16, 16), setup_lib=product).close()
    states = []
    for lib in (product, oracle):
        sim = make_sim(lib, cells=(6, 7, 8), setup_lib=product)  # partly on kept blocks
        sim.step(0.005, 3)
        if lib is product:
            tinymd.release_device_memory()
        sim.step(0.005, 20)
        states.append(tinymd.full_state(lib))
        sim.close()
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
