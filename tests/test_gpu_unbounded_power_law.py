"""A power law without an upper end (gamma_max = inf) has no grid of nodes: its
emission and absorption are 0, its Faraday terms those of the formulas
(synchrotron.py:290-311: the rotation does not see gamma_max, the conversion
grows with log(gamma_max / gamma_min)), and a thermal component beside it is
untouched."""

from __future__ import annotations

import math

import numpy as np
import pytest

import blackhole_native as bn
from blackhole_native import grrt

pytestmark = pytest.mark.gpu
FRAMES = np.array([[1e5, 10.0, 30.0, 0.3, 0.2], [1e6, 1.0, 300.0, -0.3, 1.2], [0.0, 1.0, 300.0, -0.3, 1.2]])


@pytest.mark.parametrize("n", [3, 9000])
def test_frames(n):
    f = np.resize(FRAMES, (n, 5))
    open_, closed = (bn.NonthermalPowerLawSynchrotronCoefficients(gamma_max=g) for g in (math.inf, 1e5))
    got = open_.coefficients_batch(f, 230e9)
    emits = f[:, 0] > 0
    assert np.all(got[:, :8] == 0.0) and np.all(got[~emits] == 0.0)
    assert np.array_equal(got[:, 8], closed.coefficients_batch(f, 230e9)[:, 8])
    assert np.all(np.isinf(got[emits, 9:]))
    assert np.array_equal(np.sign(got[emits, 9]), np.sign(np.cos(2 * f[emits, 4])))
    assert np.array_equal(np.sign(got[emits, 10]), np.sign(np.sin(2 * f[emits, 4])))


def test_beside_a_thermal_component():
    th = bn.ThermalSynchrotronCoefficients()
    both = bn.HybridSynchrotronCoefficients(th, bn.NonthermalPowerLawSynchrotronCoefficients(gamma_max=math.inf))
    assert np.array_equal(both.coefficients_batch(FRAMES, 230e9)[:, :8], th.coefficients_batch(FRAMES, 230e9)[:, :8])


def test_bake():
    """nan_to_num of the brick (coefficient_bricks.py:151): the largest float for +inf, 0 for -inf."""
    snap = grrt.seeded_snapshot(6, 5, 6, 0.9, 0)
    scaling = grrt.PhysicalScaling(mass_bh_g=8.54e39, distance_cm=2.57e22, rho_cgs_per_code=3.0e-18, b_gauss_per_code=25.0)
    model = bn.NonthermalPowerLawSynchrotronCoefficients(gamma_max=math.inf)
    c = bn.precompute_coefficient_bricks(snap, scaling, coeff_model=model).coeffs
    assert np.all(c[..., :8] == 0.0) and np.isin(c[..., 9:], (0.0, np.finfo(np.float32).max)).all()
