"""The batch mode's loop for steps outside the brick takes the general loop's
steps: images, step counts, statuses and Hamiltonian drifts are the same bits
as the compaction mode's, which has no such loop."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import blackhole_native as bn

pytestmark = pytest.mark.gpu

VIEWS = {
    "pole_on": dict(inclination_deg=5.0),
    "edge_on": dict(inclination_deg=90.0),
    "equator": dict(inclination_deg=89.9, h_scale=0.05, h_max=7.0),
    "south": dict(inclination_deg=160.0, phi_deg=350.0),
    "rolled": dict(inclination_deg=120.0, roll_deg=33.0, phi_deg=-725.0),
    "guard": dict(inclination_deg=60.0, horizon_guard=True),
    "small_step": dict(r_obs=60.0, fov_y_deg=30.0, h_max=0.07, max_steps=3000),
    "large_step": dict(h_scale=0.5, h_max=400.0),
    "huge_step": dict(h_scale=2.0, h_max=1e7),
    "few_steps": dict(max_steps=700),
    "one_step": dict(max_steps=1),
    "near_escape": dict(escape_radius=41.0),
    "inner_escape": dict(escape_radius=12.0, r_obs=30.0, fov_y_deg=40.0),
    "far_escape": dict(escape_radius=1e31),
    "inside": dict(r_obs=20.0, fov_y_deg=60.0, inclination_deg=45.0),
    "no_depth": dict(max_optical_depth=0.0),
    "thin": dict(max_optical_depth=1e-3),
    "spinless": dict(spin_a=0.0, inclination_deg=30.0),
    "retrograde": dict(spin_a=-0.9, inclination_deg=75.0),
}


@pytest.fixture(scope="module")
def brick():
    return bn.DeviceBrick(bn.torus_brick(40, 24, 30, spin_a=0.9, seed=2))


def _compare(brick, views, config):
    a = bn.render(brick, views, ray_outputs=True, config=config)
    b = bn.render(brick, views, ray_outputs=True, config=bn.RenderConfig(refill_min=16))
    for name in ("out", "h_drift"):
        x, y = getattr(a, name).view(torch.int32), getattr(b, name).view(torch.int32)
        assert torch.equal(x, y), name
    assert torch.equal(a.steps, b.steps) and torch.equal(a.status, b.status)
    sa, sb = a.stats(), b.stats()
    assert (sa.ray_steps, sa.brick_steps, sa.rays, sa.status) == (sb.ray_steps, sb.brick_steps, sb.rays, sb.status)
    assert (sa.max_h_drift, sa.max_h_drift_escaped) == (sb.max_h_drift, sb.max_h_drift_escaped)
    return a


@pytest.mark.parametrize("name", VIEWS)
def test_views(brick, name):
    r = _compare(brick, [bn.View(57, 41, **VIEWS[name])], bn.RenderConfig())
    if name not in ("one_step", "few_steps", "far_escape"):
        assert int((r.steps > 0).sum()) == 57 * 41


@pytest.mark.parametrize("reg_cap,blocks", [(0, 1), (80, 3), (64, 4)])
def test_all_views_in_one_launch(brick, reg_cap, blocks):
    views = [bn.View(23 + i, 17, **kw) for i, kw in enumerate(VIEWS.values())]
    _compare(brick, views, bn.RenderConfig(blocks_per_sm=blocks, reg_cap=reg_cap))
    assert np.isfinite(bn.render(brick, views).out.cpu().numpy()).all()
