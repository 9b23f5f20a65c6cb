"""A phi axis whose knots are geometric (and start above 0, as a geometric axis
does): the phi cell search has no closed form for it, so it is searched.
Images against the oracle (rel L1, the smoke tolerances: FP32 1e-3, FP64
1e-9), and the ordered sampler's time against the same call on an irregular
axis."""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import kernels
from conftest import rel_l1
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-3), ("fp64", 1e-9)])
def test_render(precision, tol):
    b = bn.torus_brick(12, 8, 24, spin_a=0.9, seed=2, dtype=np.float64)
    phi = np.geomspace(0.05, 6.0, 24).astype(np.float32).astype(np.float64)
    coeffs = b.coeffs * (0.3 + 1.7 * np.abs(np.sin(1.7 * np.arange(24))))[None, None, :, None]
    brick = bn.BrickGrid(b.r, b.theta, phi, coeffs, spin_a=0.9)
    view = bn.View(24, 16, spin_a=0.9, r_obs=55.0, inclination_deg=65.0, fov_y_deg=32.0, max_steps=900)
    img = bn.render(bn.DeviceBrick(brick, precisions=(precision,)), view, precision=precision).image().cpu().numpy()
    ov = O.make_view(spin_a=0.9, r_obs=view.r_obs, theta_obs=math.radians(view.inclination_deg), phi_obs=0.0,
                     fov_y_deg=view.fov_y_deg, roll_deg=0.0, h_scale=view.h_scale, h_min=view.h_min, h_max=view.h_max,
                     escape_radius=view.escape_radius, affine_to_length_cm=1.0, max_optical_depth=30.0, width=24,
                     height=16, x0=0, y0=0, crop_w=24, crop_h=16, max_steps=view.max_steps)
    ref = O.render(ov, coeffs, b.r, b.theta, phi, stop_at_tau=True)[0]
    assert rel_l1(img[..., 0], ref[..., 0]) <= tol


def _ms(phi):
    n = kernels.SORT_MIN_POINTS
    g = torch.Generator(device="cuda").manual_seed(1)
    f64 = dict(generator=g, device="cuda", dtype=torch.float64)
    c = torch.rand(4 * 3 * phi.size * 11, **f64)
    axes = [torch.as_tensor(a, device="cuda") for a in (np.linspace(2.0, 9.0, 4), np.linspace(0.1, 3.0, 3), phi)]
    pts = torch.rand((n, 3), **f64) * torch.tensor([7.0, 2.9, 12.0], device="cuda", dtype=torch.float64)
    pts = (pts + torch.tensor([2.0, 0.1, -6.0], device="cuda", dtype=torch.float64)).reshape(-1)
    out = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bn.sample_brick_trilinear(c, *axes, pts)
        b.record()
        b.synchronize()
        out.append(a.elapsed_time(b))
    return sorted(out[2:])[2]


def test_ordered_sampler_time():
    """8,192 knots: a walk from a wrong guess made the geometric axis 5 times as slow as the irregular one."""
    n = 8192
    irregular = 0.01 + np.cumsum(np.random.default_rng(0).uniform(0.1, 1.0, n)) * (6.0 / n)
    assert _ms(np.geomspace(0.01, 6.0, n)) < 2 * _ms(irregular)
