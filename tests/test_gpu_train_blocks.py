"""The training kernels at the edges of their 32-sample blocks.

Tolerance: a gradient entry is a sum of at most 5,000 float products in blocks
of 32 and atomic order, so two groupings differ by a few sqrt(n) roundings:
2e-5 of the layer's largest entry."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from blackhole_native import _device as dev
from blackhole_native import _lib, learned

pytestmark = pytest.mark.gpu
LAYERS = (0, 512, 576, 4672, 4736, 4800, 4801)


def _setup(n, seed=0):
    norm = np.zeros(18, dtype=np.float32)
    norm[8:16] = norm[17] = 1.0
    net = learned.StepNet.initial(norm, seed=seed)
    rows = torch.from_numpy(np.random.default_rng(seed).normal(size=(n, 9)).astype(np.float32)).cuda()
    return net, rows, torch.from_numpy(np.random.default_rng(seed + 1).permutation(n)).cuda()


def _grad(net, rows, index, first, count, shift=0):
    buf = torch.zeros(4801 + 4, dtype=torch.float32, device="cuda")
    grad, loss = buf[shift:shift + 4801], torch.zeros(1, dtype=torch.float32, device="cuda")
    _lib.check(learned._declare().bhn_mlp_grad(dev.ptr(net.params), dev.ptr(rows), dev.ptr(index), first, count,
                                               dev.ptr(grad), dev.ptr(loss), dev.stream_ptr()))
    assert float(buf[:shift].abs().sum()) == 0.0 and float(buf[shift + 4801:].abs().sum()) == 0.0
    return grad.double().cpu().numpy(), float(loss.item())


def _close(a, b):
    for lo, hi in zip(LAYERS, LAYERS[1:]):
        assert np.max(np.abs(a[lo:hi] - b[lo:hi])) <= 2e-5 * max(np.max(np.abs(b[lo:hi])), 1e-12)


@pytest.mark.parametrize("n,k", [(2, 1), (33, 32), (64, 31), (65, 33), (1000, 1), (4801, 4096)])
def test_gradients_add_up(n, k):
    """count times the mean gradient is additive over any split of the batch."""
    net, rows, index = _setup(n, n)
    whole, loss = _grad(net, rows, index, 0, n)
    a, la = _grad(net, rows, index, 0, k)
    b, lb = _grad(net, rows, index, k, n - k)
    _close(whole * n, a * k + b * (n - k))
    assert abs(loss - (la + lb)) <= 1e-4 * loss


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_gradient_buffer(shift):
    net, rows, index = _setup(500)
    _close(_grad(net, rows, index, 0, 500, shift)[0], _grad(net, rows, index, 0, 500)[0])


def test_epoch_call_takes_the_single_steps():
    L = learned._declare()
    out = []
    for whole in (True, False):
        net, rows, index = _setup(300, 5)
        g, m, v = (torch.zeros(4801, dtype=torch.float32, device="cuda") for _ in range(3))
        loss = torch.zeros(1, dtype=torch.float32, device="cuda")
        s = dev.stream_ptr()
        p = [dev.ptr(t) for t in (net.params, rows, index, g, loss, m, v)]
        if whole:
            _lib.check(L.bhn_mlp_epoch(p[0], p[1], p[2], 3, 100, p[3], p[4], p[5], p[6], 2e-3, 0.9, 0.999, 1e-8, 4, 9, s))
        else:
            for k in range(3):
                _lib.check(L.bhn_mlp_grad(p[0], p[1], p[2], 100 * k, 100, p[3], p[4], s))
                lr = 2e-3 * 0.5 * (1.0 + math.cos(math.pi * (4 + k) / 9))
                _lib.check(L.bhn_mlp_adam(p[0], p[3], p[5], p[6], lr, 0.9, 0.999, 1e-8, 5 + k, s))
        out.append(net.params.double().cpu().numpy())
    # Adam divides by |g|: entries whose gradient is rounding noise may move by a whole rate; all others agree
    moved = np.abs(out[0] - out[1])
    assert np.mean(moved > 1e-6) < 2e-3 and moved.max() <= 6.1e-3
    net, rows, index = _setup(300)
    assert L.bhn_mlp_epoch(dev.ptr(net.params), dev.ptr(rows), dev.ptr(index), 3, 100, None, None, None, None, 1e-3, 0.9,
                           0.999, 1e-8, 7, 9, dev.stream_ptr()) == 1


def test_fewer_samples_than_a_batch():
    """A batch is never larger than the samples: the same steps as with the batch given as their number."""
    rows = torch.from_numpy(np.random.default_rng(2).normal(size=(70, 9)).astype(np.float32)).cuda()
    a, b = (learned.train(rows, epochs=2, batch=n, seed=1) for n in (4096, 70))
    assert np.allclose(a.losses, b.losses, rtol=1e-4) and len(a.losses) == 2
    with pytest.raises(ValueError, match="at least one sample"):
        learned.train(rows[:0], epochs=1)
