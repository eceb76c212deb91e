"""The full-list LJ force kernels on both sides of every size at which the kernel changes (16, 8, 4 lanes
per atom or one, with and without the next gathers in flight): FP64 bit-identical to the oracle (the
pair forces are added in list order whatever the lanes), mixed within 1e-5 of the rms force, and the
mixed kernels with more FP64-path quads than their queue or marks hold."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim, rel_err

pytestmark = pytest.mark.gpu


def thermo(lib):
    t = np.zeros(4)
    assert lib.md_get_thermo(tinymd.ptr(t)) == 0
    return t


# 16 | 8 | 4 | 1 lanes: 2,048 | 2,304 and 8,112 | 8,216 and 35,912 | 36,960 atoms; one lane with the gathers
# ahead to 94,720 | without: 94,300 | 97,556; with again: 165,888
@pytest.mark.parametrize("cells", [(8, 8, 8), (8, 8, 9), (13, 13, 12), (13, 79, 2), (22, 24, 17), (20, 21, 22),
                                   (28, 29, 29), (29, 29, 29), (36, 36, 32)])
def test_fp64_bit_identical(product, oracle, cuda_device, cells):
    state = []
    for lib in (product, oracle):
        sim = make_sim(lib, cells=cells, setup_lib=product, reneigh=5)
        sim.step(0.005, 11)
        state.append(tinymd.full_state(lib))
        sim.close()
    for a, b in zip(*state):
        np.testing.assert_array_equal(a, b)


# 16 | 8 | 4 | 1 lanes: 1,008 | 1,152 and 8,112 | 9,216 and 28,880 | 30,400 atoms; gathers ahead from 300,000:
# 299,628 | 303,408
@pytest.mark.parametrize("cells", [(6, 6, 7), (6, 6, 8), (13, 13, 12), (16, 12, 12), (19, 19, 20), (20, 20, 19),
                                   (43, 42, 41), (43, 42, 42)])
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


# every pair within 1.04 sigma, so every quad has FP64-path pairs: 16, 8 and 4 lanes with up to and beyond
# 64 quads a list, one lane beyond its queue of 8, without and with the gathers ahead
@pytest.mark.parametrize("cells,cutoff", [((6, 6, 6), 2.5), ((6, 6, 6), 4.0), ((10, 10, 10), 4.0), ((17, 17, 17), 3.2),
                                          ((17, 17, 17), 4.0), ((24, 24, 24), 2.5), ((43, 42, 42), 2.5)])
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
