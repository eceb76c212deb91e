"""The DEM force kernels by size: 8, 4 or 1 lanes per grain, and the two-pass FP64 kernel for lists with
entries out of contact.  FP64 bit-identical to the oracle on both sides of every line of the rule,
with more contacts than the two-pass queue holds, mixed within the mixed form's 1e-4 of the rms
force."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim, rel_err

pytestmark = pytest.mark.gpu

DEM = (0.1, 0.1, 100.0, 0.5)


@pytest.fixture
def contact(product, oracle):
    def model(radius):
        product.md_set_dem_model(1, radius)
        oracle.oracle_set_dem_mode(1, radius)
    yield model
    product.md_set_dem_model(0, 1.0)
    oracle.oracle_set_dem_mode(0, 1.0)
    product.md_set_precision(0)


def moving(product, setup, cells):
    m, x, v, world, rank = tinymd.setup_particles(setup, cells, lib=product)
    rng = np.random.default_rng(11)
    lo, length = world[0::2], world[1::2] - world[0::2]
    x = lo + np.mod(x + rng.normal(0.0, 0.005, x.shape) - lo, length)
    return m, x, rng.normal(0.0, 0.1, x.shape), world, rank


def simulate(lib, product, particles, cutoff, steps):
    sim = make_sim(lib, benchmark="granular_gas", particles=particles, setup_lib=product, force_field="dem", dem=DEM,
                   cutoff=cutoff, reneigh=3)
    sim.step(0.001, steps)
    return sim


# gas: 8 | 4 lanes at 12,000, 4 | two-pass at 36,000, two-pass | 1 at 94,720; bed: 8 | 4 at 12,000, 4 | 1 at 72,000
@pytest.mark.parametrize("setup,cells,radius", [
    ("granular_gas", (17, 17, 16), 0.6), ("granular_gas", (18, 18, 18), 0.6), ("granular_gas", (25, 25, 25), 0.6),
    ("granular_gas", (26, 26, 26), 0.6), ("granular_gas", (36, 36, 36), 0.6), ("granular_gas", (26, 26, 26), 0.75),
    ("granular_gas", (12, 11, 10), 0.75), ("granular_gas_fcc", (18, 18, 18), 0.6),
    ("granular_gas_fcc", (20, 20, 20), 0.6), ("granular_gas_fcc", (33, 33, 32), 0.6),
    ("granular_gas_fcc", (34, 34, 34), 0.6)])
def test_fp64_bit_identical(product, oracle, cuda_device, contact, setup, cells, radius):
    contact(radius)
    particles = moving(product, setup, cells)
    state = []
    for lib in (product, oracle):
        sim = simulate(lib, product, particles, 2 * radius, 5)
        state.append(tinymd.full_state(lib))
        sim.close()
    assert np.abs(state[1][2]).max() > 0.0
    for a, b in zip(*state):
        np.testing.assert_array_equal(a, b)


# 8 | 4 lanes at 12,000 grains, 4 | 1 at 64,000
@pytest.mark.parametrize("setup,cells", [("granular_gas", (17, 17, 16)), ("granular_gas", (18, 18, 18)),
                                         ("granular_gas", (30, 30, 29)), ("granular_gas", (31, 30, 30)),
                                         ("granular_gas_fcc", (24, 24, 24))])
def test_mixed_error(product, oracle, cuda_device, contact, setup, cells):
    contact(0.6)
    product.md_set_precision(1)
    sim = simulate(product, product, moving(product, setup, cells), 1.2, 6)
    sim.force()
    f32 = tinymd.full_state(product)[2]
    product.md_set_precision(0)
    sim.force()
    f64 = tinymd.full_state(product)[2]
    sim.close()
    assert rel_err(f32, f64) <= 1e-4


@pytest.mark.parametrize("precision", [0, 1])
def test_reference_closure_stays_zero(product, cuda_device, precision):
    product.md_set_precision(precision)
    try:
        for cells in ((12, 11, 10), (20, 20, 20), (30, 30, 30)):
            sim = simulate(product, product, moving(product, "granular_gas", cells), 1.2, 2)
            assert not tinymd.full_state(product)[2].any()
            sim.close()
    finally:
        product.md_set_precision(0)
