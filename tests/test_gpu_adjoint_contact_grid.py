"""The grid that the differentiable form leaves while the contact model is set: locals and ghosts, the
ghosts' velocities included, are those of the same steps run by the step calls."""
import numpy as np
import pytest

import tinymd

pytestmark = pytest.mark.gpu

REBUILD = 4


def grid_after(product, run):
    parts = tinymd.setup_particles("default", (6, 7, 8), lib=product)
    product.md_set_dem_model(1, 0.6)
    product.md_set_ghost_mode(1)
    try:
        sim = tinymd.Simulation(product, *parts, reneigh=REBUILD)
        run(sim, np.ascontiguousarray(parts[2]))
        state = sim.arrays() + sim.ghost_arrays()
        sim.close()
    finally:
        product.md_set_dem_model(0, 1.0)
        product.md_set_ghost_mode(0)
    return state


# one, the middle and the last step of an interval, and a later interval
@pytest.mark.parametrize("steps", [1, 3, 4, 5, 10])
def test_state_after_forward(product, cuda_device, steps):
    def forward(sim, v0):
        assert product.md_adjoint_configure(steps, REBUILD, 0.002, 2.5, 0.3, 0) == 0
        assert product.md_adjoint_forward(tinymd.ptr(v0), 1.0, 1.0, tinymd.ptr(np.zeros(1))) == 0

    got = grid_after(product, forward)
    for a, b in zip(got, grid_after(product, lambda sim, v0: sim.step(0.002, steps))):
        np.testing.assert_array_equal(a, b)


def test_state_after_backward(product, cuda_device):
    """The last positions that a backward pass computes again are those before the first rebuild."""
    def both(sim, v0):
        assert product.md_adjoint_configure(10, REBUILD, 0.002, 2.5, 0.3, 0) == 0
        assert product.md_adjoint_forward(tinymd.ptr(v0), 1.0, 1.0, tinymd.ptr(np.zeros(1))) == 0
        grads = np.zeros_like(v0), np.zeros(1), np.zeros(1)
        assert product.md_adjoint_backward(*map(tinymd.ptr, grads)) == 0

    got = grid_after(product, both)
    for a, b in zip(got, grid_after(product, lambda sim, v0: sim.step(0.002, REBUILD - 1))):
        np.testing.assert_array_equal(a, b)
