"""Half lists held from both sides (the FP64 LJ kernel's) and as the reference holds them: the same
forces and sums whichever route a step takes, the reference's lists whenever they are read, and the
calls between that turn one form into the other (list reads, the mixed form, DEM, a capacity that only
the one-sided lists fit in)."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu

# a sum of at most ~80 pair forces in another order: 80 x 2^-53 of the terms' sum, whose ratio to the
# largest force stays below 1e3 here; times two for the two orders compared
RTOL = 2 * 80 * 2.0 ** -53 * 1e3


def forces(lib, sim):
    return tinymd.full_state(lib)[2][:sim.n]


def thermo(lib):
    out = np.zeros(4)
    assert lib.md_get_thermo(tinymd.ptr(out)) == 0
    return out[:3]  # energy, virial, pairs within the cutoff


def jittered(product, cells, seed=3):
    m, x, v, world, rank = tinymd.setup_particles("default", cells, lib=product)
    lo, length = world[0::2], world[1::2] - world[0::2]
    return m, lo + np.mod(x + np.random.default_rng(seed).normal(0.0, 0.08, x.shape) - lo, length), v, world, rank


@pytest.mark.parametrize("half_mode", [0, 1])
@pytest.mark.parametrize("cells,capacity", [((4, 4, 4), 0), ((7, 9, 8), 0), ((11, 12, 13), 0), ((17, 18, 19), 0),
                                            ((22, 22, 22), 0), ((7, 9, 8), 48), ((11, 12, 13), 8)])
def test_forces_and_lists_by_either_route(product, oracle, cuda_device, cells, capacity, half_mode):
    """22^3 cells: 42,592 atoms, the kernel with the next gathers in flight.  48 rows hold the
    one-sided lists of mode 0 but not the others; 8 rows neither."""
    parts = jittered(product, cells)
    product.md_set_half_mode(half_mode)
    oracle.oracle_set_half_mode(half_mode)
    product.md_set_thermo(1)
    try:
        kw = dict(half=True, particles=parts, setup_lib=product, nb_capacity=capacity, temp=None)
        p, o = make_sim(product, **kw), make_sim(oracle, **kw)
        p.step(0.001, 1)
        o.step(0.001, 1)
        f, sums = forces(product, p), thermo(product)
        fo = forces(oracle, o)
        assert np.abs(f - fo).max() <= RTOL * np.abs(fo).max()
        lists, expected = (tinymd.neighbor_lists(lib, p.n, 512) for lib in (product, oracle))
        assert sum(map(len, lists)) > 0
        assert all(np.array_equal(a, b) for a, b in zip(lists, expected))
        # the lists have turned one-sided now: the same force again
        product.md_compute_lennard_jones(True, p.cutoff, p.eps, p.sigma)
        g = forces(product, p)
        assert np.abs(f - g).max() <= RTOL * np.abs(fo).max()
        assert np.allclose(sums, thermo(product), rtol=1e-10, atol=0.0)
        p.close()
        o.close()
    finally:
        product.md_set_thermo(0)
        product.md_set_half_mode(0)
        oracle.oracle_set_half_mode(0)


def test_other_forces_over_the_same_lists(product, cuda_device):
    """Mixed half forces and a full-list force over lists built for the FP64 half kernel are those
    over the same lists after a read."""
    parts = jittered(product, (9, 10, 8))
    got = []
    for read in (False, True):
        row = []
        for call in ("mixed", "full"):
            product.md_set_half_mode(1)
            try:
                sim = make_sim(product, half=True, particles=parts, temp=None)
                if read:
                    tinymd.neighbor_lists(product, sim.n, 512)
                if call == "mixed":
                    product.md_set_precision(1)
                product.md_compute_lennard_jones(call == "mixed", sim.cutoff, sim.eps, sim.sigma)
                row.append(forces(product, sim))
                sim.close()
            finally:
                product.md_set_precision(0)
                product.md_set_half_mode(0)
        got.append(row)
    scale = np.abs(got[0][0]).max()
    assert np.abs(got[0][0] - got[1][0]).max() <= 80 * 2.0 ** -24 * 50 * scale  # FP32 sums, atomics
    assert np.array_equal(got[0][1], got[1][1])  # one-sided sums in list order
