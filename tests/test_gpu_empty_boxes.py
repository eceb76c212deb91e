"""The list build's choice of kernel in boxes with many empty cells (eight lanes per home from where the
empty cells' blocks cost more): lists equal to the oracle's, entry for entry, on both sides of the choice
for few and for many locals, in the three list modes, and after rebuilds that change it."""
import ctypes

import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu

MODES = [(False, 0), (True, 0), (True, 1)]  # half lists, half mode


def cluster(n, length):
    """n^3 cells of an fcc lattice, its sites displaced, in the corner of a cubic box"""
    a = 1.6796
    g = np.arange(n) * a
    sites = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]) * a
    x = (np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 1, 3) + sites).reshape(-1, 3)
    x = np.mod(x + np.random.default_rng(6).normal(0.0, 0.05, x.shape), length)
    return x, length


def gas(n, length):
    m = int(np.ceil(n ** (1 / 3)))
    g = (np.arange(m) + 0.5) * length / m
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n]
    return x + np.random.default_rng(6).uniform(-0.3, 0.3, x.shape) * length / m, length


def compare(product, oracle, mode, system, steps=0, **kw):
    half, half_mode = mode
    x, length = system
    world = np.array([0.0, length] * 3)
    v = np.random.default_rng(7).normal(0.0, 0.5, x.shape)
    got = []
    for lib in (product, oracle):
        set_mode = lib.oracle_set_half_mode if lib is oracle else lib.md_set_half_mode
        set_mode(half_mode)
        try:
            sim = make_sim(lib, half=half, particles=(np.ones(len(x)), x, v, world, world.copy()), temp=None, **kw)
            sim.step(0.002, steps)
            got.append(tinymd.neighbor_lists(lib, sim.n, 512))
            sim.close()
        finally:
            set_mode(0)
    assert all(np.array_equal(a, b) for a, b in zip(*got))


# clusters of 864, 4,000, 6,912 and 32,000 locals, each below and above its line; gases of 500 and 4,000
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("system", [cluster(6, 30.0), cluster(6, 90.0), cluster(10, 40.0), cluster(10, 90.0),
                                    cluster(12, 45.0), cluster(12, 100.0), cluster(20, 80.0), cluster(20, 120.0),
                                    gas(500, 20.0), gas(500, 60.0), gas(4000, 40.0), gas(4000, 60.0)])
def test_lists_equal_the_oracles(product, oracle, cuda_device, system, mode):
    compare(product, oracle, mode, system)


@pytest.mark.parametrize("system", [cluster(6, 90.0), cluster(16, 60.0), cluster(20, 80.0)])
def test_after_rebuilds(product, oracle, cuda_device, system):
    """Above 4,096 locals the first build takes the mean density, the later ones the filled cells."""
    compare(product, oracle, (False, 0), system, steps=9, reneigh=3)


def list_build_us(lib, system, builds=12):
    """Shortest of `builds` list builds, by CUDA events"""
    x, length = system
    world = np.array([0.0, length] * 3)
    sim = make_sim(lib, particles=(np.ones(len(x)), x, np.zeros_like(x), world, world.copy()), temp=None)
    kernel = [lib.md_profile_name(k) for k in range(lib.md_profile_count())].index(b"neighbor_list")
    best = np.inf
    try:
        lib.md_profile_enable(0xffff)
        for _ in range(builds):
            lib.md_profile_reset()
            sim.reneighbor()
            tinymd.check(lib)
            n, ms = ctypes.c_longlong(), ctypes.c_double()
            lib.md_profile_get(kernel, ctypes.byref(n), ctypes.byref(ms))
            best = min(best, 1e3 * ms.value / n.value)
    finally:
        lib.md_profile_enable(0)
    sim.close()
    return best


@pytest.mark.parametrize("small,large", [(gas(500, 22.0), gas(500, 140.0)), (gas(4000, 45.0), gas(4000, 140.0)),
                                         (cluster(9, 20.0), cluster(9, 140.0))])
def test_empty_cells_cost_little(product, cuda_device, small, large):
    """The same locals in 148,877 cells, most of them empty: the build is not bound by the cells (a block
    for each of them takes 82 us there, 4 to 8 times the build of the small box)."""
    assert list_build_us(product, large) <= 2.5 * list_build_us(product, small)
