"""A local with a non-finite coordinate has no neighbours (its distances compare false), so the other
atoms' forces are those of the system around it: the mixed force kernels at 16, 8 and 4 lanes per atom
and one, against the FP64 form of the same positions."""
import numpy as np
import pytest

import tinymd
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis,value", [(0, np.nan), (slice(3), np.nan), (1, -np.inf), (2, -np.inf)])
@pytest.mark.parametrize("cells", [(6, 5, 6), (13, 12, 13), (19, 19, 20), (21, 19, 21)])
def test_mixed_forces_beside_a_nonfinite_local(product, cuda_device, cells, axis, value):
    m, x, v, world, rank = tinymd.setup_particles("default", cells, lib=product)
    lo, length = world[0::2], world[1::2] - world[0::2]
    x = lo + np.mod(x + np.random.default_rng(2).normal(0.0, 0.05, x.shape) - lo, length)
    out = len(m) // 3  # inside the box: no ghosts of it
    x[out] = lo + 0.5 * length
    # at z = -inf the saturated cell index wraps to the grid's first layer (an even number of cells along
    # y), which holds no other local: the first slot
    x[out, axis] = value
    forces = []
    try:
        for precision in (1, 0):
            product.md_set_precision(precision)
            sim = tinymd.Simulation(product, m, x, v, world, rank)
            forces.append(np.delete(tinymd.full_state(product)[2], out, axis=0))
            sim.close()
    finally:
        product.md_set_precision(0)
        product.md_clear_error()  # it may lie outside the grid (5)
    assert np.isfinite(forces[1]).all()
    assert rel_err(*forces) <= 1e-5
