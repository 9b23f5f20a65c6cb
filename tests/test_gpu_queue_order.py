"""The learned and controller kernels' queue order: middle-out once there are
more packs of 32 rays than warps, slot order up to there.  A launch of few warps
and one of many take the same rays in the two orders; every output is equal."""

from __future__ import annotations

import pytest
import torch

import blackhole_native as bn
from blackhole_native import learned
from blackhole_native.render import RenderConfig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    return bn.DeviceBrick(bn.torus_brick(32, 16, 32, spin_a=0.9))


@pytest.mark.parametrize("method,sides", [("learned", [(167, 151)]), ("learned", [(160, 128)]),
                                          ("learned", [(90, 111), (33, 1), (97, 201)]), ("controller", [(211, 197)]),
                                          ("controller", [(256, 150), (1, 7)])])
def test_orders_agree(scene, method, sides):
    views = [bn.View(w, h, spin_a=0.9, inclination_deg=55.0, max_steps=4096, horizon_guard=True) for w, h in sides]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    packs = (sum(w * h for w, h in sides) + 31) // 32
    threads, many = (128, 5) if method == "learned" else (256, 4)
    warps = threads // 32 * sms
    assert warps < packs <= many * warps
    runs = []
    for blocks in (1, many):
        cfg = RenderConfig(threads, blocks, 4, 8, 32)
        if method == "learned":
            run = learned.render_learned(scene, views, learned.shipped_weights(), learned.AdaptConfig(), config=cfg,
                                         ray_outputs=True)
        else:
            run = learned.render_adaptive(scene, views, learned.AdaptConfig(), config=cfg, ray_outputs=True)
        res = run.renderer.result()
        runs.append([x.clone() for i in range(len(views))
                     for x in (res.image(i).view(torch.int32), res.per_ray("steps", i), res.per_ray("status", i))]
                    + [run.counters["steps"], run.counters["rhs_evals"]])
    for a, b in zip(*runs):
        assert torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b
