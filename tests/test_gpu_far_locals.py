"""List builds with locals far outside the box that the binning still takes: it tests only the flattened
cell index (core/grid.impala:406-411), so a far or infinite coordinate can fall into a cell of another
row, beside homes of that cell.  Every list is the oracle's: a far local has the neighbours that are
near it in space, an infinite one none, and the homes beside them keep theirs."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu

MODES = [(False, 0), (True, 0), (True, 1)]  # half lists, half mode
CUTOFF, CELL = 2.5, 2.8


def lists(lib, mode, parts):
    half, half_mode = mode
    set_mode = lib.md_set_half_mode if hasattr(lib, "md_set_half_mode") else lib.oracle_set_half_mode
    set_mode(half_mode)
    try:
        sim = make_sim(lib, half=half, cutoff=CUTOFF, particles=parts, temp=None)
        got = tinymd.neighbor_lists(lib, sim.n, 512)
        sim.close()
    finally:
        set_mode(0)
    return got


def compare(product, oracle, mode, parts, oracle_parts):
    got, expected = lists(product, mode, parts), lists(oracle, mode, oracle_parts)
    product.md_clear_error()  # locals outside the grid are reported (5)
    assert sum(map(len, got)) > 0
    assert all(np.array_equal(a, b) for a, b in zip(got, expected))
    return got


def box(world):
    """(lower corner of the grid, cells per axis) of a box of one rank (core/grid.impala:94-98)"""
    lo, hi = world[0::2] - CELL, world[1::2] + CELL
    return lo, np.floor((hi - lo + CELL / 2) / CELL).astype(int) + 1


def cluster(length, n, corner, seed=4):
    """n^3 cells of a jittered fcc lattice with its lower corner at `corner` of a cubic box"""
    a = 1.6796
    g = np.arange(n) * a
    sites = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]) * a
    x = (np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 1, 3) + sites).reshape(-1, 3) + corner
    x += np.random.default_rng(seed).normal(0.0, 0.05, x.shape)
    world = np.array([0.0, length] * 3)
    return x, world


def with_far(x, far, world):
    x = np.concatenate([x, far])
    return np.ones(len(x)), x, np.zeros_like(x), world, world.copy()


@pytest.mark.parametrize("mode", MODES)
def test_far_locals_beside_other_homes(product, oracle, cuda_device, mode):
    """Locals ~8e5 away along x whose flattened index is a cell inside the cluster."""
    x, world = cluster(196.0, 8, np.array([90.0, 90.0, 145.0]))
    lo, n = box(world)
    cell = np.unique(np.floor((x[::37] - lo) / CELL).astype(int), axis=0)
    down = cell[:, 2] - 2  # the far local's own z cell is 2; the rest of the index is along x
    far = lo + (cell + 0.5) * CELL
    far[:, 2] = lo[2] + 2.5 * CELL
    far[:, 0] += down * n[0] * n[1] * CELL
    assert np.abs(far[:, 0]).min() > 5e5 and len(x) <= 4096 - 2 * len(far)
    far = np.concatenate([far, far + [0.9, 0.2, 0.1]])  # two near each other
    parts = with_far(x, far, world)
    got = compare(product, oracle, mode, parts, parts)
    if not mode[0]:
        assert all(len(l) for l in got[len(x):])


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("axis,sign", [(0, 1), (0, -1), (1, 1), (1, -1), (2, 1), (2, -1)])
def test_infinite_locals(product, oracle, cuda_device, axis, sign, mode):
    """The oracle holds them outside the grid, where they have no neighbours either."""
    x, world = cluster(30.8, 9, np.array([5.0, 5.0, 5.0]))
    lo, n = box(world)
    assert all(k % 2 == 0 for k in n)  # the products of the saturated cell wrap into the grid
    far = x[::53].copy()
    far[:, axis] = sign * np.inf
    finite = far.copy()
    finite[:, axis] = sign * 1e6
    compare(product, oracle, mode, with_far(x, far, world), with_far(x, finite, world))
