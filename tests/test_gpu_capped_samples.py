"""A sample buffer smaller than what the controller records keeps the rows that
come first: those of the image's first rays."""

from __future__ import annotations

import pytest
import torch

import blackhole_native as bn
from blackhole_native import learned
from blackhole_native.render import RenderConfig

pytestmark = pytest.mark.gpu


def _rows(brick, view, capacity):
    samples = torch.empty((capacity, 9), dtype=torch.float32, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    learned.render_adaptive(brick, [view], learned.AdaptConfig(tol=1e-4, sample_prob=0.02), samples=samples,
                            sample_count=count, config=RenderConfig(256, 1, 4, 8, 32))
    return samples[:min(int(count.item()), capacity)].cpu().numpy(), int(count.item())


def test_capped_rows_are_the_first_rays():
    """512 x 512 rays, 37,888 of them in flight on one block per SM (74 rows of pixels): 3,000 rows come from the first 160 rows.
    Two runs record the same rows for the same rays (the hash is of the ray's slot and step)."""
    brick = bn.DeviceBrick(bn.torus_brick(32, 16, 32, spin_a=0.9))
    kw = dict(spin_a=0.9, inclination_deg=60.0, max_steps=4096, horizon_guard=True)
    top, n_top = _rows(brick, bn.View(512, 512, crop=(0, 0, 512, 160), **kw), 2_000_000)
    assert len(top) == n_top > 30_000
    capped, n_all = _rows(brick, bn.View(512, 512, **kw), 3000)
    assert len(capped) == 3000 and n_all > 2 * n_top
    known = {r.tobytes() for r in top}
    assert all(r.tobytes() in known for r in capped)
