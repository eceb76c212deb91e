"""The two list-build kernels against the oracle, entry for entry: the block per cell (well filled
cells, or few atoms) and the eight lanes per home (sparse cells, above 4,096 atoms), in the three list
modes, at the density where the choice changes, with lists that outgrow their capacity and with
locals outside the grid."""
import numpy as np
import pytest

import tinymd
from helpers import make_sim

pytestmark = pytest.mark.gpu

MODES = [(False, 0), (True, 0), (True, 1)]  # half lists, half mode


def compare(product, oracle, mode, steps=0, **kw):
    half, half_mode = mode
    got = []
    for lib in (product, oracle):
        (lib.oracle_set_half_mode if lib is oracle else lib.md_set_half_mode)(half_mode)
        try:
            sim = make_sim(lib, setup_lib=product, half=half, **kw)
            sim.step(0.002, steps)
            got.append(tinymd.neighbor_lists(lib, sim.n, 512))
            sim.close()
        finally:
            (lib.oracle_set_half_mode if lib is oracle else lib.md_set_half_mode)(0)
    assert sum(map(len, got[0])) > 0
    assert all(np.array_equal(a, b) for a, b in zip(*got))


def jittered(product, cells, seed=3):
    """An LJ lattice with displaced sites: cells and rows of uneven length."""
    m, x, v, world, rank = tinymd.setup_particles("default", cells, lib=product)
    lo, length = world[0::2], world[1::2] - world[0::2]
    x = lo + np.mod(x + np.random.default_rng(seed).normal(0.0, 0.15, x.shape) - lo, length)
    return m, x, v, world, rank


# per cell: 2.8 (sparse), 7.8 (sparse), 8.8 (dense), 18.5 (dense); 4,000 atoms always take the block per cell
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("cells,cutoff", [((11, 12, 13), 1.2), ((11, 12, 13), 1.8), ((11, 12, 13), 1.88),
                                          ((11, 12, 13), 2.5), ((10, 10, 10), 1.2), ((10, 10, 11), 1.2)])
def test_lists_equal_the_oracles(product, oracle, cuda_device, cells, cutoff, mode):
    compare(product, oracle, mode, cells=cells, cutoff=cutoff, particles=jittered(product, cells))


@pytest.mark.parametrize("setup,cells", [("granular_gas", (17, 16, 15)), ("granular_gas_fcc", (14, 15, 16))])
def test_sparse_setups_after_rebuilds(product, oracle, cuda_device, setup, cells):
    """Half-empty boxes; the third build takes its kernel from the second's count of filled cells."""
    compare(product, oracle, (False, 0), steps=21, benchmark=setup, cells=cells, cutoff=1.2, force_field="dem",
            dem=(0.1, 0.1, 100.0, 0.5), reneigh=7)


@pytest.mark.parametrize("cutoff", [1.2, 2.5])
def test_capacity_growth(product, oracle, cuda_device, cutoff):
    compare(product, oracle, (False, 0), cells=(11, 12, 13), cutoff=cutoff, nb_capacity=4,
            particles=jittered(product, (11, 12, 13)))


def test_sparse_lists_with_locals_outside_the_grid(product, oracle, cuda_device):
    m, x, v, world, rank = jittered(product, (11, 12, 13))
    x[17, 2] = world[5] + 40.0  # beyond the extended box: in no cell
    x[4000, 2] = world[4] - 40.0
    compare(product, oracle, (False, 0), cells=(11, 12, 13), cutoff=1.2, particles=(m, x, v, world, rank))
    assert product.md_last_error() == 5
    product.md_clear_error()


@pytest.mark.parametrize("mode", MODES)
def test_crowded_cells(product, oracle, cuda_device, mode):
    """Cells of ~110 atoms beside empty ones: several batches of homes, several tiles of candidates,
    lists of more entries than the buffer holds, later tiles that start inside a quad."""
    rng = np.random.default_rng(5)
    n = 1500
    world = np.array([0.0, 14.0, 0.0, 11.2, 0.0, 11.2])
    x = np.concatenate([rng.uniform(0.0, 5.6, (n, 3)), rng.uniform(0.0, 11.2, (200, 3))])
    m, v = np.ones(len(x)), np.zeros_like(x)
    compare(product, oracle, mode, cutoff=2.5, particles=(m, x, v, world, world.copy()), temp=None, nb_capacity=500)
