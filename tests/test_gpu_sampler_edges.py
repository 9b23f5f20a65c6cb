"""The sampler's batch edges (32 points a warp, 1,024 a block), its axes in and
out of shared memory, the fused input checks, and the exact Stokes step around
its switches of form, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import kernels
from oracle import oracle as O
from oracle import transfer as T

pytestmark = pytest.mark.gpu


def _scene(nr, nt, npz, n, seed):
    rng = np.random.default_rng(seed)
    rg, tg = np.cumsum(rng.uniform(0.05, 1.0, nr)), np.cumsum(rng.uniform(1e-3, 0.1, nt))
    pg = np.sort(rng.uniform(0, 2 * np.pi, npz))
    c = rng.normal(size=(nr, nt, npz, 11))
    pts = np.stack([rng.uniform(rg[0] - 0.2, rg[-1] + 0.2, n), rng.uniform(tg[0] - 0.01, tg[-1] + 0.01, n),
                    rng.uniform(-30, 30, n)], axis=1)
    if n > 4:  # knots, the last knots, phi at the wrap, whole turns
        pts[0] = rg[-1], tg[-1], pg[-1]
        pts[1] = rg[0], tg[0], pg[0] - 1e-17
        pts[2] = rg[nr // 2], tg[nt // 2], pg[0] + 2 * np.pi
        pts[3] = rg[0], tg[-1], pg[0] - 2 * np.pi
    return c, rg, tg, pg, pts


@pytest.mark.parametrize("shape,n", [((2, 2, 2), 1), ((2, 2, 2), 31), ((3, 2, 5), 33), ((9, 7, 4), 1023), ((9, 7, 4), 1025),
                                     ((5, 6, 7), 4737), ((40, 3, 4060), 2000), ((40, 3, 4053), 2000), ((3, 5, 6000), 777)])
def test_batch_edges_bit_exact(shape, n):
    c, rg, tg, pg, pts = _scene(*shape, n, n)
    dev = [torch.as_tensor(x, device="cuda") for x in (c, rg, tg, pg, pts)]
    got = bn.sample_brick_trilinear(*dev).cpu().numpy().reshape(n, 11)
    assert np.array_equal(got, O.sample_brick_trilinear(c, rg, tg, pg, pts), equal_nan=True)
    ini = np.random.default_rng(n).normal(size=(n, 4))
    for policy in ("nan", "initial", "zero"):
        got = bn.sample_and_step_stokes(*dev, 0.3, torch.as_tensor(ini, device="cuda"), policy).cpu().numpy()
        assert np.array_equal(got.reshape(n, 4), O.sample_and_step_stokes(c, rg, tg, pg, pts, 0.3, ini, policy),
                              equal_nan=True)


@pytest.mark.parametrize("kind", ["uniform", "geometric", "random", "one_gap"])
def test_cell_order_on_every_axis_kind(kind):
    """The key kernel's closed-form cells: large point sets on uniform, geometric and irregular axes equal the
    input-order kernel's results."""
    rng = np.random.default_rng(7)
    n = kernels.SORT_MIN_POINTS + 77
    if kind == "uniform":
        rg, tg, pg = np.linspace(-3.0, 40.0, 37), np.linspace(0.0, 3.0, 19), np.linspace(0.0, 6.2, 23)
    elif kind == "geometric":
        rg, tg, pg = np.geomspace(1e-3, 1e3, 37), np.geomspace(0.1, 3.0, 19), np.geomspace(0.01, 6.0, 23)
    elif kind == "random":
        rg, tg, pg = (np.cumsum(rng.uniform(1e-6, 1.0, m)) * s for m, s in ((37, 1.0), (19, 0.1), (23, 0.2)))
    else:
        rg, tg, pg = np.r_[np.arange(36.0), 1e6], np.r_[0.0, np.linspace(2.0, 3.0, 18)], np.linspace(1.0, 1.5, 23)
    c = torch.as_tensor(rng.normal(size=(37, 19, 23, 11)).ravel(), device="cuda")
    pts = rng.uniform([rg[0], tg[0], -20.0], [rg[-1], tg[-1], 20.0], (n, 3))
    pts[:5000, 0] = rng.choice(rg, 5000)
    pts[5000:9000, 1] = rng.choice(tg, 4000)
    pts[9000:12000, 2] = rng.choice(pg, 3000) + 2 * np.pi * rng.integers(-3, 4, 3000)
    axes = [torch.as_tensor(g, device="cuda") for g in (rg, tg, pg)]
    dp = torch.as_tensor(pts.ravel(), device="cuda")
    big = bn.sample_brick_trilinear(c, *axes, dp)
    half = 3 * (n // 2)
    small = torch.cat([bn.sample_brick_trilinear(c, *axes, dp[:half]), bn.sample_brick_trilinear(c, *axes, dp[half:])])
    assert n // 2 < kernels.SORT_MIN_POINTS
    assert torch.equal(big.view(torch.int64), small.view(torch.int64))


@pytest.mark.parametrize("what,message", [("r", "r grid must contain only finite"), ("tinc", "theta grid must be strictly"),
                                          ("phi", "phi grid must contain only finite"), ("coeffs", "coeffs must contain only"),
                                          ("points", "points must contain only finite"), ("initial", "initial must contain only finite"),
                                          ("r+points", "r grid must contain only finite"), ("len", "initial must contain either 4")])
@pytest.mark.parametrize("n", [50, kernels.SORT_MIN_POINTS])
def test_device_inputs_are_checked(what, message, n):
    c, rg, tg, pg, pts = _scene(6, 5, 8, n, 1)
    ini = np.zeros(5 if what == "len" else 4)
    if "r" in what.split("+"):
        rg[3] = np.nan
    if what == "tinc":
        tg[2] = tg[1]
    if what == "phi":
        pg[-1] = np.inf
    if what == "coeffs":
        c[5, 4, 7, 10] = -np.inf
    if "points" in what:
        pts[n - 1, 2] = np.nan
    if what == "initial":
        ini[3] = np.inf
    dev = [torch.as_tensor(x, device="cuda") for x in (c, rg, tg, pg, pts)]
    with pytest.raises(ValueError, match=message):
        bn.sample_and_step_stokes(*dev, 0.1, torch.as_tensor(ini, device="cuda"))
    if what not in ("initial", "len"):
        with pytest.raises(ValueError, match=message):
            bn.sample_brick_trilinear(*dev)


@pytest.mark.parametrize("norm", [0.0, 1e-9, 1 / 256, 1 / 64, 1 / 16, 0.25, 0.5, 0.99, 1.0, 1.01, 2.0, 2.01, 3.99, 4.0, 4.01, 30.0])
def test_exact_step_forms(norm):
    """||K ds|| at the series' term counts and step counts and at the change to squaring.  Both forms drop less than
    2^-56 and round some 20 products: 1e-13 of the step's size (|S| + |j| ds) e^norm covers both and the oracle's."""
    rng = np.random.default_rng(int(norm * 1000) + 1)
    n = 200
    c = rng.normal(size=(n, 11))
    K = np.abs(c[:, 4:])
    size = np.max([K[:, 0] + K[:, 1] + K[:, 2] + K[:, 3], K[:, 0] + K[:, 1] + K[:, 4] + K[:, 6],
                   K[:, 0] + K[:, 2] + K[:, 4] + K[:, 5], K[:, 0] + K[:, 3] + K[:, 5] + K[:, 6]], axis=0)
    ds = 0.7
    c[:, 4:] *= (norm / (size * ds))[:, None]
    s = rng.normal(size=(n, 4))
    got = bn.stokes_exact_brick(torch.as_tensor(c.ravel(), device="cuda"), ds, torch.as_tensor(s.ravel(), device="cuda"))
    want = np.array([T.stokes_step_exact(s[i], c[i], ds) for i in range(n)])
    scale = (np.abs(s).max(1) + np.abs(c[:, :4]).max(1) * ds) * np.exp(norm)
    assert np.all(np.abs(got.cpu().numpy().reshape(n, 4) - want) <= 1e-13 * scale[:, None])


def test_cells_are_checked_in_the_same_pass():
    c, s = torch.ones(11 * 300, dtype=torch.float64, device="cuda"), torch.zeros(1200, dtype=torch.float64, device="cuda")
    for step in (bn.stokes_rk2_brick, bn.stokes_exact_brick):
        bad = c.clone()
        bad[11 * 299 + 10] = float("inf")
        with pytest.raises(ValueError, match="coeffs must contain only finite"):
            step(bad, 0.1, s)
        bad = s.clone()
        bad[-1] = float("nan")
        with pytest.raises(ValueError, match="initial must contain only finite"):
            step(c, 0.1, bad)
        with pytest.raises(ValueError, match="either 4 values"):
            step(c, 0.1, s[:8])
