"""Which results keep their bits when a job is cut differently: bricks (any cut
of the snapshot, any cell count), images (any crop), frame batches on either
side of the length from which the power law's nodes are summed in groups.
Across that length frames agree to 1e-11 (each coefficient is a sum of positive
terms, each with a few roundings of an exponent of at most ~600)."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import _device as dev
from blackhole_native import _lib, grrt
from test_gpu_synchrotron_sums import GROUPED, _close, _frames

pytestmark = pytest.mark.gpu
SCALING = grrt.PhysicalScaling(mass_bh_g=8.54e39, distance_cm=2.57e22, rho_cgs_per_code=3.0e-18, b_gauss_per_code=25.0)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_a_brick_of_few_cells_is_a_part_of_the_larger_one(dtype):
    snap = grrt.seeded_snapshot(24, 16, 40, 0.9, 0)  # 15,360 cells; shells of 640
    whole = bn.precompute_coefficient_bricks(snap, SCALING, dtype=dtype).coeffs
    for a, b in ((0, 1), (5, 8), (12, 24), (0, 13)):
        part = SimpleNamespace(r=snap.r[a:b], theta=snap.theta, phi=snap.phi, rho=snap.rho[a:b], theta_e=snap.theta_e[a:b],
                               b_con=snap.b_con[a:b], spin_a=snap.spin_a)
        out = bn.synchrotron.precompute_device_coefficients(part, SCALING, dtype=dtype)[3].cpu().numpy()
        assert np.array_equal(out, whole[a:b])


def test_a_crop_of_few_rays_is_a_part_of_the_image(monkeypatch):
    snap = grrt.DeviceSnapshot(grrt.seeded_snapshot(24, 12, 24, 0.9, 0))
    cfg = grrt.PolarizedRenderConfig(width=12, height=8, max_steps=1500)
    lib, seen = grrt._declare(), []

    class Seen:
        bhn_grrt_scratch_bytes = lib.bhn_grrt_scratch_bytes

        @staticmethod
        def bhn_grrt_render_scratch(*a):
            seen.append(a)
            return lib.bhn_grrt_render_scratch(*a)

    monkeypatch.setattr(grrt, "_declare", lambda: Seen)
    image = grrt.render_stokes_image_device(cfg, snap, SCALING)
    assert float(image[2:6, 3:9, 0].abs().sum()) > 0.0
    v = seen[0][7]._obj
    scratch = torch.empty(1 << 22, dtype=torch.float64, device="cuda")  # the first call's went back with its return
    tables = bn.synchrotron.table_scratch(seen[0][8]._obj, scratch.device)
    sp = (dev.ptr(scratch) + 255) & ~255
    for x0, y0, w, h in ((3, 2, 1, 1), (4, 3, 3, 2), (5, 2, 2, 4), (2, 2, 9, 1)):
        v.x0, v.y0, v.crop_w, v.crop_h = x0, y0, w, h
        out = torch.empty((h, w, 4), dtype=torch.float64, device="cuda")
        a = list(seen[0])
        a[10:17] = [sp, 8 * scratch.numel() - 256, dev.ptr(tables), tables.numel(), dev.ptr(out), None, dev.stream_ptr()]
        _lib.check(lib.bhn_grrt_render_scratch(*a))
        assert torch.equal(out.view(torch.int64), image[y0:y0 + h, x0:x0 + w].contiguous().view(torch.int64))


def test_frames_around_the_grouped_length():
    f = _frames(2 * GROUPED + 5, 3)
    for model in (bn.HybridSynchrotronCoefficients(), bn.NonthermalPowerLawSynchrotronCoefficients()):
        def run(n):
            return model.coefficients_batch(f[:n], 230e9)

        below, above = run(GROUPED - 1), run(GROUPED)
        assert np.array_equal(below[:33], run(33)) and np.array_equal(below[:1], run(1))
        assert np.array_equal(above, run(2 * GROUPED + 5)[:GROUPED])
        assert _close(above[:-1], below, 1e-11)
