"""The synchrotron models' tables in caller memory: sizes without a GPU; on the
GPU the package takes them from torch (the library's own pool is left alone),
and the forms with and without scratch give the same bits."""

from __future__ import annotations

import ctypes
import math
import subprocess
import sys

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import _device as dev
from blackhole_native import _lib, grrt
from blackhole_native import synchrotron as syn
from tests.conftest import PKG_ROOT

Hybrid, Thermal, Power = (bn.HybridSynchrotronCoefficients, bn.ThermalSynchrotronCoefficients,
                          bn.NonthermalPowerLawSynchrotronCoefficients)


def _bytes(model):
    syn._table_bytes.cache_clear()
    m = syn.model_struct(model, 230e9, syn._UNIT_SCALING)
    return syn._table_bytes(syn._table_values(m))


@pytest.mark.parametrize("pitch", [1, 2, 3, 16, 17, 33, 64])
@pytest.mark.parametrize("gamma_n,lo,hi", [(2, 10.0, 1e5), (224, 10.0, 1e5), (4096, 1.0, 1.001), (16, 1e-300, 1e300),
                                           (224, 10.0, math.inf)])
def test_sizes(pitch, gamma_n, lo, hi):
    """Bounded for every accepted model, an unbounded power law among them (whose plan has no node, and so no table)."""
    nt = Power(pitch_nodes=pitch, gamma_grid_size=gamma_n, gamma_min=lo, gamma_max=hi)
    for other in (1, 16, 64):
        both = _bytes(Hybrid(Thermal(pitch_nodes=other), nt))
        assert 0 < both <= 9_000_000 and both % 256 == 0
    assert _bytes(nt) == 256 if hi == math.inf else 256 < _bytes(nt) <= 9_000_000


@pytest.mark.parametrize("model", [Power(gamma_min=5.0, gamma_max=5.0), Power(pitch_nodes=65), Thermal(gamma_grid_size=1)])
def test_refused_models(model):
    assert _bytes(model) == -1


def _frames(n):
    rng = np.random.default_rng(n)
    f = np.stack([10.0 ** rng.uniform(3, 7, n), 10.0 ** rng.uniform(-1.5, 2.5, n), 10.0 ** rng.uniform(-2, 4, n),
                  rng.uniform(-1, 1, n), rng.uniform(-2, 2, n)], axis=1)
    return torch.from_numpy(f).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 8191, 8192])
@pytest.mark.parametrize("model", [Hybrid(), Thermal(), Power(), Power(gamma_max=math.inf)])
def test_scratch_and_pool_forms_agree(model, n):
    f = _frames(n)
    want = model.coefficients_batch(f, 230e9)  # the scratch form
    got = torch.empty_like(want)
    m = syn.model_struct(model, 230e9, syn._UNIT_SCALING)
    _lib.check(syn._declare_frames().bhn_synchrotron_coefficients(dev.ptr(f), n, ctypes.byref(m), dev.ptr(got), dev.stream_ptr()))
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))


@pytest.mark.gpu
def test_scratch_is_checked():
    f, out = _frames(40), torch.empty((40, 11), dtype=torch.float64, device="cuda")
    m = syn.model_struct(Hybrid(), 230e9, syn._UNIT_SCALING)
    buf = syn.table_scratch(m, out.device)
    fn = syn._declare_frames().bhn_synchrotron_coefficients_scratch
    for p, n in ((dev.ptr(buf), 100_000), (dev.ptr(buf) + 16, buf.numel()), (None, buf.numel())):
        assert fn(dev.ptr(f), 40, ctypes.byref(m), dev.ptr(out), p, n, dev.stream_ptr()) == 1
        assert b"model scratch" in _lib.lib().bhn_last_error()


POOL = """
import ctypes, sys
import numpy as np, torch
import blackhole_native as bn
from blackhole_native import _device as dev, _lib, grrt, synchrotron as syn
f = torch.ones((64, 5), dtype=torch.float64, device="cuda")
model = bn.HybridSynchrotronCoefficients()
snap = grrt.seeded_snapshot(8, 6, 8, 0.9, 0)
scaling = grrt.PhysicalScaling(mass_bh_g=8.54e39, distance_cm=2.57e22, rho_cgs_per_code=3.0e-18, b_gauss_per_code=25.0)
model.coefficients_batch(f, 230e9)
bn.precompute_coefficient_bricks(snap, scaling)
grrt.render_stokes_image_device(grrt.PolarizedRenderConfig(width=4, height=2, max_steps=50), grrt.DeviceSnapshot(snap), scaling)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
out = torch.empty((64, 11), dtype=torch.float64, device="cuda")
m = syn.model_struct(model, 230e9, syn._UNIT_SCALING)
_lib.check(syn._declare_frames().bhn_synchrotron_coefficients(dev.ptr(f), 64, ctypes.byref(m), dev.ptr(out), dev.stream_ptr()))
print("grew", before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.gpu
def test_the_package_leaves_the_librarys_pool_alone():
    """In a fresh process the pool's first allocation comes with the first call of a form without scratch."""
    run = subprocess.run([sys.executable, "-c", POOL], env={**__import__("os").environ, "PYTHONPATH": str(PKG_ROOT)},
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr
    assert int(run.stdout.split("grew")[1]) > 0


@pytest.mark.gpu
def test_grrt_pool_form_agrees():
    snap = grrt.DeviceSnapshot(grrt.seeded_snapshot(16, 8, 16, 0.9, 0))
    scaling = grrt.PhysicalScaling(mass_bh_g=8.54e39, distance_cm=2.57e22, rho_cgs_per_code=3.0e-18, b_gauss_per_code=25.0)
    cfg = grrt.PolarizedRenderConfig(width=12, height=6, max_steps=800)
    want = grrt.render_stokes_image_device(cfg, snap, scaling)
    lib = grrt._declare()
    calls = []

    class Pool:  # the call's own arguments without the tables' memory
        bhn_grrt_scratch_bytes = lib.bhn_grrt_scratch_bytes

        @staticmethod
        def bhn_grrt_render_scratch(*a):
            calls.append(1)
            return lib.bhn_grrt_render(*a[:12], *a[14:])

    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(grrt, "_declare", lambda: Pool)
        got = grrt.render_stokes_image_device(cfg, snap, scaling)
    assert calls == [1] and torch.equal(got.view(torch.int64), want.view(torch.int64))


def test_sizes_do_not_depend_on_what_was_planned_before():
    """Each pitch count's plan is kept; counts in any order, one component or two, give the sizes of a fresh process."""
    models = [Hybrid(Thermal(pitch_nodes=a), Power(pitch_nodes=b)) for a in (64, 2, 16, 1) for b in (3, 64, 16)]
    first = [_bytes(m) for m in models]
    assert [_bytes(m) for m in reversed(models)] == first[::-1]
    code = ("import blackhole_native as bn\nfrom blackhole_native import synchrotron as s\n"
            "m = s.model_struct(bn.HybridSynchrotronCoefficients(bn.ThermalSynchrotronCoefficients(pitch_nodes=2),"
            " bn.NonthermalPowerLawSynchrotronCoefficients(pitch_nodes=64)), 230e9, s._UNIT_SCALING)\n"
            "print(s._table_bytes(s._table_values(m)))")
    fresh = subprocess.run([sys.executable, "-c", code], env={**__import__("os").environ, "PYTHONPATH": str(PKG_ROOT)},
                           capture_output=True, text=True, timeout=300)
    assert int(fresh.stdout) == _bytes(Hybrid(Thermal(pitch_nodes=2), Power(pitch_nodes=64)))
