"""The guiding network's kernels where their tiles and groups begin and end:
one row, one below, at and above a 128-row tile, every CTA with one tile of
its first group only, the second group's first tile, a third round; outputs
that are not 16-byte aligned. Against the same fp32 torch network as
test_gpu_guide.py, with its tolerances."""
import numpy as np
import pytest

from test_gpu_guide import LAYERS, TOL, flat_grads, mixture_nll, torch_forward, torch_net, torch_params

pytestmark = pytest.mark.gpu

TILE, SMS = 128, 152
ROWS = [1, TILE - 1, TILE, TILE + 1, SMS * TILE, SMS * TILE + 1, 2 * SMS * TILE + 1, 3 * SMS * TILE - 5]


@pytest.mark.parametrize("n", ROWS)
def test_forward_and_backward(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.25, 15592).astype(np.float32)
    gpu.guide_set_params(p)
    x = rng.normal(0, 1, (n, 7)).astype(np.float32)
    dout = rng.normal(0, 1, (n, 40)).astype(np.float32)
    dx, dd = torch.tensor(x, device="cuda:0"), torch.tensor(dout, device="cuda:0")
    outs = [torch.full((n * 40 + 4,), float("nan"), device="cuda:0") for _ in range(2)]
    grads = [torch.full((15592,), float("nan"), device="cuda:0") for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(2):
        gpu.guide_forward_dev(dx.data_ptr(), n, outs[k].data_ptr() + 4 * k)
        gpu.guide_backward_dev(dx.data_ptr(), dd.data_ptr(), n, grads[k].data_ptr())
    a, b = outs[0][:n * 40].cpu().numpy(), outs[1][1:n * 40 + 1].cpu().numpy()
    assert np.array_equal(a, b)  # the same values at an address that is not a multiple of 16
    assert np.isnan(outs[0][n * 40:].cpu().numpy()).all() and np.isnan(outs[1][n * 40 + 1:].cpu().numpy()).all()
    want = torch_forward(p, x)
    assert np.abs(a.reshape(n, 40) - want).max() <= TOL * np.abs(want).max()
    g = grads[0].cpu().numpy()
    assert np.array_equal(g, grads[1].cpu().numpy())  # partials are added in a fixed order
    layers = torch_params(p, True)
    (torch_net(layers, torch.tensor(x)) * torch.tensor(dout)).sum().backward()
    want, o = flat_grads(layers), 0
    for kin, kout in LAYERS:
        for size in (kin * kout, kout):
            w = want[o:o + size]
            # dZ is rounded to fp16 on its way down the layers; one row has no other rows' rounding to average with
            assert np.abs(g[o:o + size] - w).max() <= 2e-2 * max(np.abs(w).max(), 1e-12)
            o += size


@pytest.mark.parametrize("n", ROWS)
def test_loss_of_a_step(gpu, n):
    import torch
    rng = np.random.default_rng(n + 1)
    gpu.guide_init(seed=5)
    p = gpu.guide_params()
    x = rng.normal(0, 1, (n, 7)).astype(np.float32)
    d = rng.normal(0, 1, (n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    w = rng.exponential(1.0, n).astype(np.float32)
    dx, ddir, dw = (torch.tensor(a, device="cuda:0") for a in (x, d, w))
    torch.cuda.synchronize()
    loss = gpu.guide_train_step_dev(dx.data_ptr(), ddir.data_ptr(), dw.data_ptr(), n, 1e-4)
    want = mixture_nll(torch_net(torch_params(p), torch.tensor(x)), torch.tensor(d), torch.tensor(w)).item()
    assert abs(loss - want) <= 1e-3 * abs(want)
    moved = np.abs(gpu.guide_params() - p)
    assert np.isfinite(moved).all() and moved.max() <= 1.05e-4 and (moved > 0).mean() > 0.3
