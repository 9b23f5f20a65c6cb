"""The tabulated sums behind the synchrotron integrals (bhn_synchrotron.cuh):
pitch averages of any node count, the power law's node groups, frame batches
of any length, against the oracle and against each other.

Tolerance: every coefficient is a sum of positive terms, each with a few
roundings of an exponent of at most ~600 (1e-13 relative) and a tabulation
error below that, so 1e-11 relative where the coefficient is a normal number."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import blackhole_native as bn
from oracle import synchrotron as S

pytestmark = pytest.mark.gpu
GROUPED = 8192  # frames from which the power law's nodes are taken in groups


def _frames(n, seed):
    rng = np.random.default_rng(seed)
    f = np.empty((n, 5))
    f[:, 0] = 10.0 ** rng.uniform(3, 7, n)
    f[:, 1] = 10.0 ** rng.uniform(-1.5, 2.5, n)
    f[:, 2] = 10.0 ** rng.uniform(-2, 4, n)
    f[:, 3] = rng.uniform(-1, 1, n)
    f[:, 4] = rng.uniform(-2, 2, n)
    return f


def _oracle(frames, nu, th, nt):
    out = np.zeros((len(frames), 11))
    for i, (n_e, te, b, cos, chi) in enumerate(frames):
        if th is not None:
            out[i] += S.thermal(n_e, te, b, chi, nu, dict(vars(th)), cos)
        if nt is not None:
            out[i] += S.nonthermal(n_e, te, b, chi, nu, dict(vars(nt)), cos)
    return out


def _close(got, want, rtol=1e-11):
    # the rotated components (Q, U pairs) are held to their pair's size
    scale = np.abs(want)
    for q, u in ((1, 2), (5, 6), (9, 10)):
        scale[:, q] = scale[:, u] = np.hypot(want[:, q], want[:, u])
    ok = scale >= 1e-290
    return np.all(np.abs(got - want)[ok] <= rtol * scale[ok]) and np.all(np.abs(got[~ok]) < 1e-280)


@pytest.mark.parametrize("pitch", [1, 2, 3, 16, 17, 33, 63, 64])
@pytest.mark.parametrize("gamma_n", [2, 7, 33])
def test_node_counts_against_the_oracle(pitch, gamma_n):
    th = bn.ThermalSynchrotronCoefficients(gamma_grid_size=gamma_n, pitch_nodes=pitch)
    nt = bn.NonthermalPowerLawSynchrotronCoefficients(gamma_grid_size=gamma_n + 1, pitch_nodes=max(1, pitch - 1))
    f = _frames(12, pitch)
    got = bn.HybridSynchrotronCoefficients(th, nt).coefficients_batch(f, 230e9)
    assert _close(got, _oracle(f, 230e9, th, nt))


@pytest.mark.parametrize("pitch,gamma_n,p,lo,hi", [(16, 224, 3.5, 10.0, 1e5), (16, 225, 1.0, 1.0, 1e3), (5, 7, 2.2, 3.0, 30.0),
                                                   (16, 8, 2.5, 1.0, 1e6), (64, 257, 0.5, 50.0, 1e4), (1, 4096, 6.0, 2.0, 1e7)])
def test_grouped_nodes_equal_single_nodes(pitch, gamma_n, p, lo, hi):
    """A batch large enough for node groups against small batches of the same frames, and the oracle."""
    nt = bn.NonthermalPowerLawSynchrotronCoefficients(p=p, gamma_min=lo, gamma_max=hi, gamma_grid_size=gamma_n,
                                                      pitch_nodes=pitch)
    f = _frames(GROUPED, gamma_n)
    big = nt.coefficients_batch(f, 86e9)
    pick = np.r_[0:40, GROUPED - 40:GROUPED]
    assert _close(big[pick], nt.coefficients_batch(f[pick], 86e9))
    assert _close(big[pick[::8]], _oracle(f[pick[::8]], 86e9, None, nt))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 3551, 3553, 7105])
def test_a_frame_does_not_depend_on_its_batch(n):
    """Batches around the frames-per-warp steps; empty frames among them."""
    f = _frames(n, 3)
    f[::5, 0] = 0.0
    model = bn.HybridSynchrotronCoefficients()
    got = model.coefficients_batch(f, 230e9)
    one = np.concatenate([model.coefficients_batch(f[i:i + 1], 230e9) for i in {0, n // 2, n - 1}])
    assert np.array_equal(got[sorted({0, n // 2, n - 1})], one[np.argsort(list({0, n // 2, n - 1}))])
    assert np.all(got[::5] == 0.0)


def test_frames_under_graph_capture():
    """The call's tables are the graph's own memory when it is captured; replays see new frames."""
    model = bn.HybridSynchrotronCoefficients()
    fd = torch.from_numpy(_frames(500, 1)).cuda()
    model.coefficients_batch(fd, 230e9)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = model.coefficients_batch(fd, 230e9)
    for seed in (1, 2):
        fd.copy_(torch.from_numpy(_frames(500, seed)))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), model.coefficients_batch(_frames(500, seed), 230e9))
