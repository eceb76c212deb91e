"""The adjoint's step and size rules: every shape of the last list interval (one kernel per step inside
an interval, a checkpoint between two) against FP64 autograd of the all-pairs trajectory, the lanes
per atom of the product kernel on both sides of each size where they change against FP64 autograd
over a pair list, and the state that a backward pass leaves."""
import numpy as np
import pytest
import torch

import tinymd
from tinymd import adjoint
from test_gpu_adjoint import adjoint_grads, allpairs_lj, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,reneigh", [(1, 1), (1, 5), (2, 1), (5, 5), (6, 5), (7, 3), (10, 5), (11, 4)])
def test_intervals(product, cuda_device, steps, reneigh):
    sim, parts, v0 = setup(product, (4, 4, 4))
    try:
        adjoint.configure(product, steps=steps, reneigh=reneigh, dt=0.005, precision=0, shifted_energy=True)
        grads = [adjoint_grads(product, v0) for _ in range(2)]
    finally:
        sim.close()
    m, x, _, world, _ = parts
    box = torch.tensor(world[1::2] - world[0::2], dtype=torch.float64)
    v = torch.tensor(v0, requires_grad=True)
    e, s = (torch.tensor(1.0, dtype=torch.float64, requires_grad=True) for _ in range(2))
    loss = allpairs_lj.trajectory_loss(torch.tensor(x), v, e, s, box, 0.005, steps, shifted=True)
    loss.backward()
    for got, gv, ge, gs in grads:
        assert got == pytest.approx(float(loss.detach()), rel=1e-10)
        assert ge == pytest.approx(float(e.grad), rel=1e-8)
        assert gs == pytest.approx(float(s.grad), rel=1e-8)
        assert np.max(np.abs(gv - v.grad.numpy())) <= 1e-8 * float(v.grad.abs().max())
    np.testing.assert_array_equal(grads[0][1], grads[1][1])


def pair_list_gradients(x0, v0, length, steps, reach=2.8, rc=2.5, dt=0.005):
    """Loss and gradients by autograd over the pairs within `reach` at x0 (all pairs that can come
    inside rc in the few steps), in FP64 torch."""
    dev = torch.device("cuda")
    x = torch.tensor(x0, device=dev)
    box = torch.tensor(length, device=dev)
    pairs = []
    for b in range(0, len(x0), 512):
        d = x[b:b + 512, None] - x[None]
        d = d - box * torch.round(d / box)
        i, j = torch.nonzero((d * d).sum(-1) < reach * reach, as_tuple=True)
        pairs.append(torch.stack([i + b, j])[:, i + b != j])
    i, j = torch.cat(pairs, 1)
    v = torch.tensor(v0, device=dev, requires_grad=True)
    eps, sigma = (torch.tensor(1.0, dtype=torch.float64, device=dev, requires_grad=True) for _ in range(2))

    def terms(y):
        d = y[i] - y[j]
        d = d - box * torch.round(d / box)
        r2 = (d * d).sum(-1)
        inside = r2 < rc * rc
        sr2 = torch.where(inside, 1.0 / r2, torch.zeros_like(r2))
        sr6 = sr2 ** 3 * sigma ** 6
        return d, inside, sr2, sr6

    def force(y):
        d, _, sr2, sr6 = terms(y)
        return torch.zeros_like(y).index_add_(0, i, (48.0 * eps * sr6 * (sr6 - 0.5) * sr2)[:, None] * d)

    y, w, f = x, v, force(x)
    for _ in range(steps):
        w = w + 0.5 * dt * f
        y = y + dt * w
        f = force(y)
        w = w + 0.5 * dt * f
    _, inside, _, sr6 = terms(y)
    cut6 = (sigma / rc) ** 6
    energy = 0.5 * (4.0 * eps * (sr6 * (sr6 - 1.0) - inside * (cut6 * (cut6 - 1.0)))).sum()
    loss = ((y - x) ** 2).sum() / len(x0) + energy / len(x0)
    g = torch.autograd.grad(loss, [v, eps, sigma])
    return float(loss.detach()), g[0].cpu().numpy(), float(g[1]), float(g[2])


# 32 | 16 | 8 | 4 lanes: 2,916 | 3,600 and 5,760 | 6,336 and 11,760 | 12,544 atoms
@pytest.mark.parametrize("cells", [(9, 9, 9), (10, 10, 9), (12, 12, 10), (12, 12, 11), (14, 14, 15), (14, 14, 16)])
def test_lanes(product, cuda_device, cells):
    sim, parts, v0 = setup(product, cells)
    try:
        adjoint.configure(product, steps=3, reneigh=2, dt=0.005, precision=0, shifted_energy=True)
        loss, gv, ge, gs = adjoint_grads(product, v0)
    finally:
        sim.close()
    world = parts[3]
    want = pair_list_gradients(parts[1], v0, world[1::2] - world[0::2], 3)
    assert loss == pytest.approx(want[0], rel=1e-10)
    assert ge == pytest.approx(want[2], rel=1e-8)
    assert gs == pytest.approx(want[3], rel=1e-8)
    assert np.max(np.abs(gv - want[1])) <= 1e-8 * np.max(np.abs(want[1]))


def test_state_after_backward(product, cuda_device):
    """The grid is left at the first interval's last recomputed step: the driver's own loop gives it."""
    sim, parts, v0 = setup(product, (5, 6, 7))
    try:
        adjoint.configure(product, steps=9, reneigh=6, dt=0.005, precision=0)
        adjoint_grads(product, v0)
        left = tinymd.full_state(product)
    finally:
        sim.close()
    m, x, _, world, rank = parts
    product.md_set_ghost_mode(1)
    try:
        run = tinymd.Simulation(product, m, x, v0, world, rank, reneigh=100)
        run.step(0.005, 5)
        want = tinymd.full_state(product)
        run.close()
    finally:
        product.md_set_ghost_mode(0)
    for a, b in zip(left, want):
        np.testing.assert_array_equal(a, b)
