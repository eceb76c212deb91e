"""The LJ force kernels that share an atom between 2 to 16 lanes, on both sides of every size at
which the number of lanes changes: FP64 bit-identical to the oracle (the pair forces are added in
list order whatever the lanes), mixed within 1e-5 of the rms force, and the mixed kernels' redo of
an atom whose FP64-path quads overflow the queue."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim, rel_err

pytestmark = pytest.mark.gpu


def thermo(lib):
    t = np.zeros(4)
    assert lib.md_get_thermo(tinymd.ptr(t)) == 0
    return t


# 16 | 8 | 4 | 1 lanes: 2,048 | 2,304 and 6,864 | 7,488 and 38,808 | 40,656 atoms
@pytest.mark.parametrize("cells", [(8, 8, 8), (8, 8, 9), (13, 11, 12), (12, 13, 12), (21, 21, 22), (21, 22, 22)])
def test_fp64_bit_identical(product, oracle, cuda_device, cells):
    state = []
    for lib in (product, oracle):
        sim = make_sim(lib, cells=cells, setup_lib=product, reneigh=5)
        sim.step(0.005, 11)
        state.append(tinymd.full_state(lib))
        sim.close()
    for a, b in zip(*state):
        np.testing.assert_array_equal(a, b)


# 16 | 8 | 4 | 2 | 1 lanes: 2,048 | 2,304 and 16,384 | 17,408 and 48,668 | 50,784 and 81,648 | 84,672 atoms
@pytest.mark.parametrize("cells", [(8, 8, 8), (8, 8, 9), (16, 16, 16), (16, 16, 17), (23, 23, 23), (23, 23, 24),
                                   (27, 27, 28), (27, 28, 28)])
def test_mixed_error(product, cuda_device, cells):
    """Forces and sums of the mixed form on the state after 21 steps against the FP64 form's."""
    product.md_set_precision(1)
    product.md_set_thermo(1)
    try:
        sim = make_sim(product, cells=cells, setup_lib=product, reneigh=5)
        sim.step(0.005, 21)
        out = []
        for precision in (1, 0):
            product.md_set_precision(precision)
            sim.force()
            product.md_final_integration(0.0)
            out.append((tinymd.full_state(product)[2], thermo(product)))
        sim.close()
    finally:
        product.md_set_precision(0)
        product.md_set_thermo(0)
    (f32, t32), (f64, t64) = out
    assert rel_err(f32, f64) <= 1e-5
    assert t32[2] == t64[2]
    np.testing.assert_allclose(t32[[0, 3]], t64[[0, 3]], rtol=1e-6)


# every pair within 1.04 sigma: 8, 4, 2 and 1 lanes with more than 8 queued quads per lane
@pytest.mark.parametrize("cells,cutoff", [((10, 10, 10), 4.0), ((17, 17, 17), 3.2), ((24, 24, 24), 2.5),
                                          ((28, 28, 28), 2.5)])
def test_mixed_queue_overflow(product, cuda_device, cells, cutoff):
    product.md_set_precision(1)
    try:
        m, x, v, world, rank = tinymd.setup_particles("default", cells, lib=product)
        x = x + np.random.default_rng(1).normal(0.0, 0.05, x.shape)
        sim = tinymd.Simulation(product, m, x, v, world, rank, cutoff=cutoff, sigma=cutoff, nb_capacity=320)
        f32 = tinymd.full_state(product)[2]
        product.md_set_precision(0)
        sim.force()
        f64 = tinymd.full_state(product)[2]
        sim.close()
    finally:
        product.md_set_precision(0)
    assert rel_err(f32, f64) <= 1e-5
