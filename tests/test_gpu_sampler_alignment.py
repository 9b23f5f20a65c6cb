"""The cell-ordered sampler's wide point reads and result writes, chosen by the
arrays' alignment: every alignment gives the input-order kernel's bits."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import _device as dev, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 1025, 4737])
@pytest.mark.parametrize("pts_offset,out_offset", [(0, 0), (3, 0), (0, 2), (1, 2), (2, 4)])
def test_alignments_agree(n, pts_offset, out_offset):
    rng = np.random.default_rng(n)
    nr, nt, npz = 9, 7, 6
    rg, tg, pg = np.linspace(1.0, 9.0, nr), np.linspace(0.2, 2.9, nt), np.linspace(0.0, 5.9, npz)
    axes = [torch.as_tensor(g, device="cuda") for g in (rg, tg, pg)]
    c = torch.as_tensor(rng.normal(size=nr * nt * npz * 11), device="cuda")
    pts = torch.zeros(3 * n + pts_offset, dtype=torch.float64, device="cuda")[pts_offset:]
    pts.copy_(torch.as_tensor(rng.uniform([0.8, 0.1, -9.0], [9.2, 3.0, 9.0], (n, 3)).ravel()))
    ini = torch.as_tensor(rng.normal(size=4 * n), device="cuda")
    L = _lib.lib()
    need = int(L.bhn_sample_sort_scratch_bytes(n, nr * nt * npz))
    scratch = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    base = (dev.ptr(scratch) + 255) & ~255
    got = []
    for ordered in (False, True):
        out = torch.full((4 * n + out_offset + 4,), 7.0, dtype=torch.float64, device="cuda")
        args = (dev.ptr(c), dev.ptr(axes[0]), nr, dev.ptr(axes[1]), nt, dev.ptr(axes[2]), npz, dev.ptr(pts), n, 0.3,
                dev.ptr(ini), ini.numel(), 0, dev.ptr(out) + 8 * out_offset)
        if ordered:
            _lib.check(L.bhn_sample_and_step_stokes_sorted(*args, base, need, dev.stream_ptr()))
        else:
            _lib.check(L.bhn_sample_and_step_stokes(*args, dev.stream_ptr()))
        torch.cuda.synchronize()
        assert bool((out[:out_offset] == 7.0).all()) and bool((out[out_offset + 4 * n:] == 7.0).all())
        got.append(out[out_offset:out_offset + 4 * n].view(torch.int64).clone())
    assert torch.equal(*got)


@pytest.mark.parametrize("per_warp", [4, 8, 16])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_points_per_warp(per_warp, extra):
    """Around the point counts where a warp's share changes: a call equals its points in calls of other shares."""
    n = torch.cuda.get_device_properties(0).multi_processor_count * 32 * per_warp + extra
    rng = np.random.default_rng(n)
    nr, nt, npz = 9, 7, 6
    axes = [torch.as_tensor(g, device="cuda") for g in
            (np.linspace(1.0, 9.0, nr), np.linspace(0.2, 2.9, nt), np.linspace(0.0, 5.9, npz))]
    c = torch.as_tensor(rng.normal(size=nr * nt * npz * 11), device="cuda")
    pts = torch.as_tensor(rng.uniform([0.8, 0.1, -9.0], [9.2, 3.0, 9.0], (n, 3)).ravel(), device="cuda")
    whole = bn.sample_brick_trilinear(c, *axes, pts)
    cuts = [0, 7, n // 5, n // 2, n]
    parts = torch.cat([bn.sample_brick_trilinear(c, *axes, pts[3 * a:3 * b]) for a, b in zip(cuts, cuts[1:])])
    assert torch.equal(whole.view(torch.int64), parts.view(torch.int64))
