"""The sampler's points per warp (4, 8, 16, 32 by the set's size and the brick's):
on either side of each line the same bits as the oracle, or for a brick too
large for L2 as smaller sets of the same points."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import blackhole_native as bn
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _lines():
    return torch.cuda.get_device_properties(0).multi_processor_count * 32


@pytest.mark.parametrize("points", [2, 6, 12])
@pytest.mark.parametrize("more", [0, 1])
def test_lines_bit_exact(points, more):
    n = points * _lines() + more
    rng = np.random.default_rng(points)
    rg, tg, pg = np.geomspace(1.5, 60.0, 9), np.linspace(0.05, 3.1, 7), np.linspace(0.0, 6.0, 8)
    c = rng.normal(size=(9, 7, 8, 11))
    pts = rng.uniform([1.0, 0.0, -9.0], [61.0, 3.2, 9.0], (n, 3))
    ini = rng.normal(size=(n, 4))
    dev = [torch.as_tensor(x, device="cuda") for x in (c, rg, tg, pg, pts)]
    got = bn.sample_brick_trilinear(*dev).cpu().numpy().reshape(n, 11)
    assert np.array_equal(got, O.sample_brick_trilinear(c, rg, tg, pg, pts), equal_nan=True)
    got = bn.sample_and_step_stokes(*dev, 0.3, torch.as_tensor(ini, device="cuda"), "zero").cpu().numpy().reshape(n, 4)
    assert np.array_equal(got, O.sample_and_step_stokes(c, rg, tg, pg, pts, 0.3, ini, "zero"), equal_nan=True)


@pytest.mark.parametrize("points,more", [(12, 1), (16, 0), (16, 1)])
def test_large_brick(points, more):
    n = points * _lines() + more
    g = torch.Generator(device="cuda").manual_seed(points)
    f64 = dict(generator=g, device="cuda", dtype=torch.float64)
    c = torch.rand(128 * 80 * 128 * 11, **f64)  # 115 MB
    axes = [torch.as_tensor(a, device="cuda") for a in (np.geomspace(1.5, 60.0, 128), np.linspace(0.05, 3.1, 80), np.linspace(0.0, 6.2, 128))]
    pts = (torch.rand((n, 3), **f64) * torch.tensor([58.0, 3.0, 12.0], device="cuda", dtype=torch.float64) + 1.6).reshape(-1)
    whole = bn.sample_brick_trilinear(c, *axes, pts)
    parts = torch.cat([bn.sample_brick_trilinear(c, *axes, p) for p in pts.split(3 * 5003)])
    assert torch.equal(whole.view(torch.int64), parts.view(torch.int64))
