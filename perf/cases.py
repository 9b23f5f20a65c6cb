"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call, ``run`` makes one pass through the public entry points, ``work`` says
what a pass cannot do without and ``exact`` gives the 64-bit result where one
exists.  Kinds of case:

* ``points``  the plugin micro-kernels ``sample_brick_trilinear`` (op "sample")
  and ``sample_and_step_stokes`` (op "step"): from the reference's own call
  with lists (a few dozen points) to millions of points on device tensors.
* ``cells``   ``stokes_rk2_brick`` / ``stokes_exact_brick`` over many cells.
* ``frames``  a synchrotron model's ``coefficients_batch`` on device frames.
* ``bake``    ``precompute_coefficient_bricks``: host snapshot in, host brick out.
* ``bricks``  the reference's brick renderer (RK4, FP64) on a device brick.
* ``grrt``    the physical polarized renderer on a device snapshot.
* ``image``   a prepared ``Renderer`` of one view (plain RK2, FP32 or FP64).
* ``views``   a prepared ``Renderer`` of many uneven views, per-ray outputs on.
* ``steps``   the adaptive loops: ``render_learned`` and ``render_adaptive``.
* ``train``   the step network's training (forward, backward, Adam).
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "blackhole-sim_b200"))

import blackhole_native as bn  # noqa: E402
from blackhole_native import accelerated, grrt, learned, synchrotron  # noqa: E402

TWO_PI = 2.0 * math.pi
SCALING = dict(mass_bh_g=8.54e39, distance_cm=2.57e22, rho_cgs_per_code=3.0e-18, b_gauss_per_code=25.0)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference benchmark's own call: an 8x6x8 brick and 64 points, all passed as lists
        {"name": "points_list_64", "kind": "points", "op": "step", "points": 64, "nr": 8, "nt": 6, "np": 8,
         "host": True, "policy": "nan"},
        # a batch of ray samples through a small brick, tensors in and out
        {"name": "points_100k", "kind": "points", "op": "sample", "points": 100_003, "nr": 64, "nt": 33, "np": 60,
         "host": False, "policy": "nan"},
        # a whole wavefront's samples through the headline brick (738 MB in float64)
        {"name": "points_12M", "kind": "points", "op": "step", "points": 12_582_912, "nr": 256, "nt": 128, "np": 256,
         "host": False, "policy": "nan"},
        # the exact Stokes step of every cell of a mid-size brick, each with its own Stokes vector
        {"name": "cells_exact_2M", "kind": "cells", "op": "exact", "cells": 2_000_003, "own_initial": True,
         "ds": 0.05},
        # plasma frames sampled along rays by a caller's own tracer
        {"name": "frames_30k", "kind": "frames", "frames": 30_011, "model": "hybrid", "ghz": 230.0},
        # a GRMHD snapshot baked to the float32 brick the renderers take
        {"name": "bake_2M", "kind": "bake", "nr": 160, "nt": 96, "np": 160, "dtype": "float32", "ghz": 230.0},
        # the reference's default brick image
        {"name": "bricks_160x90", "kind": "bricks", "width": 160, "height": 90, "nr": 128, "nt": 64, "np": 128,
         "exact_step": False, "wide": False, "spin": 0.9375, "incl": 65.0},
        # the reference's default physical image
        {"name": "grrt_160x90", "kind": "grrt", "width": 160, "height": 90, "nr": 64, "nt": 32, "np": 64,
         "exact_step": False, "spin": 0.9375, "incl": 65.0},
        # the headline image: 1024 x 1024 rays, 4096 RK2 steps, 256 x 128 x 256 brick
        {"name": "image_1024", "kind": "image", "width": 1024, "height": 1024, "r_obs": 1000.0, "spin": 0.9375,
         "incl": 17.0, "max_steps": 4096, "precision": "fp32", "guard": False, "nr": 256, "nt": 128, "np": 256},
        # a batch of uneven views (a parameter sweep) in one launch
        {"name": "views_12", "kind": "views", "count": 12, "side_lo": 64, "side_hi": 512, "mix": 0, "nr": 128,
         "nt": 64, "np": 128},
        # an image by the learned step
        {"name": "learned_512", "kind": "steps", "method": "learned", "side": 512, "spin": 0.9375, "incl": 30.0,
         "tol": 1e-4, "nr": 128, "nt": 64, "np": 128},
        # one epoch of the step network's training on recorded steps
        {"name": "train_64k", "kind": "train", "samples": 65_536, "batch": 4096, "epochs": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _brick_shape(rng, hi):
    return {"nr": _log_int(rng, 6, hi), "nt": _log_int(rng, 5, hi // 2), "np": _log_int(rng, 6, hi)}


def draw(rng):
    kind = rng.choice(["points", "points", "cells", "frames", "bake", "bricks", "grrt", "image", "image", "views",
                       "steps", "train"])
    if kind == "points":
        host = rng.random() < 0.25
        n = _log_int(rng, 1, 2000) if host else _log_int(rng, 50, 12_000_000)
        c = {"op": rng.choice(["sample", "step"]), "points": n, "host": host,
             "policy": rng.choice(["nan", "initial", "zero"])}
        c.update(_brick_shape(rng, 16 if host else 256))
        if c["op"] == "sample":
            c["policy"] = "nan"  # the sampler has no policy: rejected points are NaN rows
    elif kind == "cells":
        c = {"op": rng.choice(["rk2", "exact"]), "cells": _log_int(rng, 1000, 8_000_000),
             "own_initial": rng.random() < 0.5, "ds": rng.choice([0.02, 0.05, 0.5, 2.0])}
    elif kind == "frames":
        c = {"frames": _log_int(rng, 1, 100_000), "model": rng.choice(["hybrid", "thermal", "powerlaw"]),
             "ghz": rng.choice([43.0, 86.0, 230.0, 345.0])}
    elif kind == "bake":
        c = {"nr": _log_int(rng, 8, 160), "nt": _log_int(rng, 8, 96), "np": _log_int(rng, 8, 160),
             "dtype": rng.choice(["float32", "float64"]), "ghz": rng.choice([86.0, 230.0])}
    elif kind == "bricks":
        w = _log_int(rng, 40, 640)
        c = {"width": w, "height": max(3, int(w * rng.uniform(0.5, 1.0))), "exact_step": rng.random() < 0.3,
             "wide": rng.random() < 0.3, "spin": round(rng.uniform(0.0, 0.95), 4),
             "incl": round(rng.uniform(20.0, 85.0), 2)}
        c.update(_brick_shape(rng, 128))
    elif kind == "grrt":
        w = _log_int(rng, 16, 160)
        c = {"width": w, "height": max(2, int(w * rng.uniform(0.4, 0.56))), "exact_step": rng.random() < 0.5,
             "spin": round(rng.uniform(0.0, 0.95), 4), "incl": round(rng.uniform(30.0, 80.0), 2)}
        c.update(_brick_shape(rng, 64))
    elif kind == "image":
        fp64 = rng.random() < 0.3
        w = _log_int(rng, 24, 384 if fp64 else 1024)
        c = {"width": w, "height": max(2, int(w * rng.uniform(0.5, 1.0))), "r_obs": rng.choice([55.0, 1000.0]),
             "spin": round(rng.uniform(0.0, 0.998), 4), "incl": round(rng.uniform(5.0, 85.0), 2),
             "max_steps": _log_int(rng, 512, 8192), "precision": "fp64" if fp64 else "fp32",
             "guard": rng.random() < 0.5}
        c.update(_brick_shape(rng, 256))
    elif kind == "views":
        c = {"count": rng.randint(2, 40), "side_lo": 16, "side_hi": rng.randint(64, 512),
             "mix": rng.randint(0, 10**6)}
        c.update(_brick_shape(rng, 128))
    elif kind == "steps":
        c = {"method": rng.choice(["learned", "controller"]), "side": _log_int(rng, 48, 1024),
             "spin": round(rng.uniform(0.0, 0.998), 4), "incl": round(rng.uniform(5.0, 85.0), 2),
             "tol": rng.choice([2e-5, 1e-4])}
        c.update(_brick_shape(rng, 128))
    else:
        c = {"samples": _log_int(rng, 4096, 200_000), "batch": rng.choice([1000, 2048, 4096]), "epochs": 1}
    return {"kind": kind, **c}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grids(case, spin, single):
    """r log-spaced from 1.05 r_+ to 40 M, theta at cell centres of (0, pi), phi uniform on [0, 2 pi)."""
    r = np.geomspace(1.05 * (1.0 + math.sqrt(1.0 - spin * spin)), 40.0, case["nr"])
    th = math.pi * (np.arange(case["nt"]) + 0.5) / case["nt"]
    ph = np.linspace(0.0, TWO_PI, case["np"], endpoint=False)
    return [g.astype(np.float32).astype(np.float64) if single else g for g in (r, th, ph)]


def _torus(grids, gen, dtype):
    """A torus's 11 transfer coefficients on the grid: the package's synthetic scene, drawn on the device."""
    r, th, _ = (torch.as_tensor(g, device="cuda") for g in grids)
    shape = tuple(g.size for g in grids)
    out = torch.empty(shape + (11,), dtype=dtype, device="cuda")
    dens = torch.exp(-((r[:, None] - 8.0) ** 2) / 8.0 - 4.0 * torch.cos(th)[None, :] ** 2)
    fj = torch.tensor([1.0, 0.2, 0.1, 0.02], dtype=torch.float64, device="cuda")
    rot = torch.tensor([0.5, 0.1, 0.05], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // (shape[1] * shape[2] * 11))
    for a in range(0, shape[0], step):
        b = min(shape[0], a + step)
        ln = torch.exp(0.05 * torch.randn((b - a,) + shape[1:] + (11,), generator=gen, device="cuda",
                                          dtype=torch.float64))
        u = torch.rand((b - a,) + shape[1:] + (3,), generator=gen, device="cuda", dtype=torch.float64) + 0.5
        d = dens[a:b, :, None, None]
        j = d * fj * ln[..., 0:4]
        out[a:b, ..., 0:4] = j
        out[a:b, ..., 4:8] = 0.1 * j * ln[..., 4:8]
        out[a:b, ..., 8:11] = d * rot * u * ln[..., 8:11]
    return out


def _points_inputs(case, seed):
    gen = _gen(seed)
    grids = _grids(case, 0.9375, False)
    coeffs = _torus(grids, gen, torch.float64).reshape(-1)
    n = case["points"]
    u = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    r, th, _ = grids
    # about one point in thirty lies outside the brick's r range, phi runs over several turns
    lo = torch.tensor([r[0] - 0.4, th[0], -4.0 * math.pi], dtype=torch.float64, device="cuda")
    hi = torch.tensor([r[-1] + 0.8, th[-1], 4.0 * math.pi], dtype=torch.float64, device="cuda")
    pts = lo + u * (hi - lo)
    ini = torch.tensor([0.01, 0.001, -0.002, 0.0005], dtype=torch.float64, device="cuda")
    return grids, coeffs, pts, ini


def _cells_inputs(case, seed):
    gen = _gen(seed)
    n = case["cells"]
    r = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    dens = torch.exp(-8.0 * (r - 0.4) ** 2)[:, None]
    ln = torch.exp(0.05 * torch.randn((n, 11), generator=gen, device="cuda", dtype=torch.float64))
    f = torch.tensor([1.0, 0.2, 0.1, 0.02, 0.1, 0.02, 0.01, 0.002, 0.5, 0.1, 0.05], dtype=torch.float64, device="cuda")
    c = (dens * f * ln).reshape(-1)
    if case["own_initial"]:
        ini = torch.rand((n, 4), generator=gen, device="cuda", dtype=torch.float64)
        ini[:, 1:] = 0.3 * (ini[:, 1:] - 0.5)
        ini = ini.reshape(-1)
    else:
        ini = torch.tensor([0.3, 0.02, -0.01, 0.005], dtype=torch.float64, device="cuda")
    return c, case["ds"], ini


def _frames_inputs(case, seed):
    gen = _gen(seed)
    n = case["frames"]
    u = torch.rand((n, 5), generator=gen, device="cuda", dtype=torch.float64)
    f = torch.empty_like(u)
    f[:, 0] = 10.0 ** (3.0 + 4.0 * u[:, 0])            # n_e [cm^-3]
    f[:, 1] = 10.0 ** (-0.5 + 2.3 * u[:, 1])           # Theta_e 0.3 .. 63
    f[:, 2] = 10.0 ** (2.0 * u[:, 2])                  # B 1 .. 100 G
    f[:, 3] = 2.0 * u[:, 3] - 1.0                      # cos of the pitch to the line of sight
    f[:, 4] = math.pi * (u[:, 4] - 0.5)                # EVPA
    return f


def _model(name):
    if name == "thermal":
        return synchrotron.ThermalSynchrotronCoefficients()
    if name == "powerlaw":
        return synchrotron.NonthermalPowerLawSynchrotronCoefficients()
    return synchrotron.HybridSynchrotronCoefficients()


def _snapshot(case, seed, spin):
    """A GRMHD-like snapshot on the host: torus density, log-uniform Theta_e, Gaussian field, slow rotation."""
    gen = _gen(seed)
    grids = _grids(case, spin, False)
    r, th, _ = (torch.as_tensor(g, device="cuda") for g in grids)
    shape = tuple(g.size for g in grids)
    rho = torch.exp(-((r[:, None, None] - 8.0) ** 2) / 8.0 - 4.0 * torch.cos(th)[None, :, None] ** 2)
    rho = rho * torch.exp(0.2 * torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))
    te = torch.exp(math.log(60.0) * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64))
    b = torch.randn(shape + (4,), generator=gen, device="cuda", dtype=torch.float64)
    u = torch.zeros(shape + (4,), dtype=torch.float64, device="cuda")
    u[..., 0] = 1.0
    u[..., 3] = 0.5 * r[:, None, None] ** -1.5
    rho, te, b, u = (t.cpu().numpy() for t in (rho, te, b, u))
    return grrt.Snapshot(r=grids[0], theta=grids[1], phi=grids[2], rho=rho, theta_e=te, pressure=rho * te, b_con=b,
                         u_con=u, spin_a=spin)


class _Spin:
    def __init__(self, a):
        self.spin_a = a


class _HostBrick:
    def __init__(self, grids, coeffs):
        self.r, self.theta, self.phi = grids
        self.coeffs = coeffs


def _device_brick(case, spin, seed, precision="fp32"):
    grids = _grids(case, spin, True)
    coeffs = _torus(grids, _gen(seed), torch.float32)
    return bn.DeviceBrick.from_device_coeffs(*grids, coeffs, spin_a=spin, precisions=(precision,))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "points":
        grids, coeffs, pts, ini = _points_inputs(case, seed)
        if case["host"]:
            args = [coeffs.tolist(), *(g.tolist() for g in grids), pts.reshape(-1).tolist(), ini.tolist()]
        else:
            args = [coeffs, *(torch.as_tensor(g, device="cuda") for g in grids), pts.reshape(-1), ini]
        return {"case": case, "args": args}
    if kind == "cells":
        c, ds, ini = _cells_inputs(case, seed)
        return {"case": case, "args": (c, ds, ini)}
    if kind == "frames":
        return {"case": case, "model": _model(case["model"]), "frames": _frames_inputs(case, seed)}
    if kind == "bake":
        return {"case": case, "snapshot": _snapshot(case, seed, 0.9375), "scaling": grrt.PhysicalScaling(**SCALING)}
    if kind == "bricks":
        grids = _grids(case, case["spin"], True)
        coeffs = _torus(grids, _gen(seed), torch.float64 if case["wide"] else torch.float32).cpu().numpy()
        cfg = accelerated.AcceleratedRenderConfig(
            width=case["width"], height=case["height"],
            camera=grrt.LocalCamera.from_degrees(r=55.0, inclination_degrees=case["incl"], fov_y_degrees=32.0),
            transfer=grrt.PolarizedTransferConfig(use_exact_matrix_step=case["exact_step"]))
        return {"case": case, "cfg": cfg, "spin": _Spin(case["spin"]),
                "bricks": accelerated.DeviceBricks(_HostBrick(grids, coeffs))}
    if kind == "grrt":
        cfg = grrt.PolarizedRenderConfig(
            width=case["width"], height=case["height"],
            camera=grrt.LocalCamera.from_degrees(r=55.0, inclination_degrees=case["incl"], fov_y_degrees=32.0),
            transfer=grrt.PolarizedTransferConfig(use_exact_matrix_step=case["exact_step"]))
        return {"case": case, "cfg": cfg, "scaling": grrt.PhysicalScaling(**SCALING),
                "snapshot": grrt.DeviceSnapshot(_snapshot(case, seed, case["spin"]))}
    if kind == "image":
        view = bn.View(case["width"], case["height"], spin_a=case["spin"], r_obs=case["r_obs"],
                       inclination_deg=case["incl"], max_steps=case["max_steps"], horizon_guard=case["guard"],
                       **({} if case["r_obs"] > 100.0 else {"fov_y_deg": 32.0}))
        db = _device_brick(case, case["spin"], seed, case["precision"])
        return {"case": case, "renderer": bn.Renderer(db, [view], precision=case["precision"])}
    if kind == "views":
        n = case["count"]
        sides = np.random.default_rng(case["mix"]).integers(case["side_lo"], case["side_hi"] + 1, size=n)
        rng = np.random.default_rng(seed)
        views = [bn.View(int(s), int(s), spin_a=float(a), inclination_deg=float(i), max_steps=int(m))
                 for s, a, i, m in zip(sides, rng.uniform(0.0, 0.998, n), rng.uniform(5.0, 85.0, n),
                                       rng.integers(512, 8193, size=n))]
        db = _device_brick(case, 0.998, seed)
        return {"case": case, "renderer": bn.Renderer(db, views, ray_outputs=True)}
    if kind == "steps":
        view = bn.View(case["side"], case["side"], spin_a=case["spin"], inclination_deg=case["incl"], max_steps=8192,
                       horizon_guard=True)
        return {"case": case, "view": view, "brick": _device_brick(case, case["spin"], seed),
                "net": learned.shipped_weights()}
    gen = _gen(seed)
    n = case["samples"]
    x = torch.randn((n, 9), generator=gen, device="cuda", dtype=torch.float32)
    x[:, 0] = 2.5 + 1.5 * x[:, 0]
    x[:, 1] = torch.tanh(x[:, 1])
    x[:, 4] = 0.998 * torch.sigmoid(x[:, 4])
    x[:, 7] = -12.0 + 8.0 * torch.sigmoid(x[:, 7])
    x[:, 8] = 0.4 * x[:, 0] - torch.square(x[:, 2]) * 0.2 + 0.5 * torch.sin(x[:, 6]) + 0.1 * x[:, 8]
    return {"case": case, "samples": x, "seed": seed % 7}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "points":
        c, r, th, ph, pts, ini = state["args"]
        if case["op"] == "sample":
            out = bn.sample_brick_trilinear(c, r, th, ph, pts)
        else:
            out = bn.sample_and_step_stokes(c, r, th, ph, pts, 0.05, ini, case["policy"])
        return np.asarray(out) if case["host"] else out
    if kind == "cells":
        step = bn.stokes_rk2_brick if case["op"] == "rk2" else bn.stokes_exact_brick
        return step(*state["args"])
    if kind == "frames":
        return state["model"].coefficients_batch(state["frames"], case["ghz"] * 1e9)
    if kind == "bake":
        return bn.precompute_coefficient_bricks(state["snapshot"], state["scaling"], case["ghz"] * 1e9,
                                                dtype=case["dtype"]).coeffs
    if kind == "bricks":
        return accelerated.render_stokes_image_bricks_device(state["cfg"], state["spin"], state["bricks"])
    if kind == "grrt":
        return grrt.render_stokes_image_device(state["cfg"], state["snapshot"], state["scaling"])
    if kind == "image":
        return state["renderer"].launch().out
    if kind == "views":
        res = state["renderer"].launch()
        return {"stokes": res.out, "steps": res.steps, "status": res.status}
    if kind == "steps":
        if case["method"] == "learned":
            m = learned.render_learned(state["brick"], [state["view"]], state["net"], learned.AdaptConfig())
        else:
            m = learned.render_adaptive(state["brick"], [state["view"]], learned.AdaptConfig(tol=case["tol"]))
        return {"stokes": m.image(), "counters": m.counters}
    net = learned.train(state["samples"], epochs=case["epochs"], batch=case["batch"], seed=state["seed"])
    # the loss is accumulated in float32 on the device
    return {"params": net.params, "loss": torch.tensor(net.losses, dtype=torch.float32)}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    cells = case.get("nr", 0) * case.get("nt", 0) * case.get("np", 0)
    if kind == "points":
        n = case["points"]
        touched = min(8 * n, cells)  # cells whose 88 bytes some point needs
        out = 88 if case["op"] == "sample" else 32
        return {"bytes": 88 * touched + n * (24 + out), "flops": n * (8 * 11 * 3 + (100 if case["op"] == "step" else 0))}
    if kind == "cells":
        n = case["cells"]
        return {"bytes": n * (88 + 32 + (32 if case["own_initial"] else 0)),
                "flops": n * (100 if case["op"] == "rk2" else 600)}
    # a synchrotron evaluation: two kernels at every Lorentz-factor node and distinct pitch angle, a few operations each
    nodes = {"hybrid": 416, "thermal": 192, "powerlaw": 224}[case.get("model", "hybrid")]
    if kind == "frames":
        return {"bytes": case["frames"] * 128, "flops": case["frames"] * nodes * 8 * 2 * 4}
    if kind == "bake":
        return {"bytes": cells * (48 + 11 * {"float64": 8, "float32": 4}[case["dtype"]]),
                "flops": cells * nodes * 8 * 2 * 4}
    if kind == "bricks":
        n = case["width"] * case["height"]
        return {"bytes": cells * 11 * (8 if case["wide"] else 4) + 32 * n, "flops": n * 1500 * 577}
    if kind == "grrt":
        n = case["width"] * case["height"]
        return {"bytes": cells * 88 + 32 * n, "flops": n * (1500 * 577 + 1200 * nodes * 8 * 2 * 4)}
    if kind == "image":
        n = case["width"] * case["height"]
        steps = min(case["max_steps"], 1300 if case["r_obs"] > 100.0 else 350)
        b = 4 if case["precision"] == "fp32" else 8
        return {"bytes": cells * 12 * b + 4 * b * n, "flops": n * steps * 213}
    if kind == "views":
        sides = np.random.default_rng(case["mix"]).integers(case["side_lo"], case["side_hi"] + 1, size=case["count"])
        n = int((sides ** 2).sum())
        return {"bytes": cells * 48 + 21 * n, "flops": n * 1300 * 213}
    if kind == "steps":
        n = case["side"] ** 2
        return {"bytes": cells * 48 + 16 * n, "flops": n * 250 * 450}
    n = case["samples"] // case["batch"] * case["batch"] * case["epochs"]
    return {"bytes": 36 * n + 4 * 4801 * 5 * (n // case["batch"]), "flops": n * 3 * 2 * (8 * 64 + 64 * 64 + 64)}


# ------------------------------------------------------------------ 64-bit results
def _bracket(g, x):
    i = (torch.searchsorted(g, x, right=True) - 1).clamp(0, g.numel() - 2)
    return i, (x - g[i]) / (g[i + 1] - g[i])


def _exact_samples(grids, coeffs, pts):
    r, th, ph = (torch.as_tensor(g, device="cuda") for g in grids)
    nt, npz = th.numel(), ph.numel()
    inside = (pts[:, 0] >= r[0]) & (pts[:, 0] <= r[-1]) & (pts[:, 1] >= th[0]) & (pts[:, 1] <= th[-1])
    ir, wr = _bracket(r, pts[:, 0])
    it, wt = _bracket(th, pts[:, 1])
    p = torch.remainder(pts[:, 2] - ph[0], TWO_PI) + ph[0]
    ip = (torch.searchsorted(ph, p, right=True) - 1).clamp(0, npz - 1)
    ip1 = (ip + 1) % npz
    wp = (p - ph[ip]) / (torch.where(ip1 > ip, ph[ip1], ph[0] + TWO_PI) - ph[ip])
    c = coeffs.view(-1, 11)
    out = torch.zeros((pts.shape[0], 11), dtype=torch.float64, device="cuda")
    for dr in (0, 1):
        for dt in (0, 1):
            for q, w in ((ip, 1.0 - wp), (ip1, wp)):
                at = ((ir + dr) * nt + it + dt) * npz + q
                out += ((wr if dr else 1.0 - wr) * (wt if dt else 1.0 - wt) * w)[:, None] * c[at]
    out[~inside] = math.nan
    return out, inside


def _matrix(c):
    ai, aq, au, av, rv, rq, ru = c[:, 4:].unbind(1)
    k = torch.stack([ai, aq, au, av, aq, ai, rv, -ru, au, -rv, ai, rq, av, ru, -rq, ai], dim=1)
    return k.view(-1, 4, 4)


def _exact_rk2(c, ds, s):
    k = _matrix(c)
    rhs = lambda x: c[:, :4] - torch.einsum("nij,nj->ni", k, x)  # noqa: E731
    return s + ds * rhs(s + 0.5 * ds * rhs(s))


def _kernel_table():
    """log x, log F, log G of the 256-entry synchrotron kernel table; K_{2/3} by the trapezoid rule (DLMF 10.32.9)."""
    xs = np.geomspace(1.0e-8, 1.0e3, 256)
    F = 1.25 * xs ** (1.0 / 3.0) * np.exp(-xs) * (648.0 + xs * xs) ** (1.0 / 12.0)
    G = np.empty_like(xs)
    for i, x in enumerate(xs):
        h = min(0.02, 0.25 / math.sqrt(x))
        t = np.arange(0.0, math.acosh(1.0 + 750.0 / x) + h, h)
        y = np.exp(-x * np.cosh(t)) * np.cosh(2.0 / 3.0 * t)
        G[i] = x * h * (0.5 * y[0] + y[1:].sum())
    return [torch.as_tensor(np.log(v), device="cuda") for v in (xs, np.maximum(F, 1e-300), np.maximum(G, 1e-300))]


def _exact_component(n_e, te, b, nu, thermal, table):
    """Pitch-averaged j_I and j_Q of one distribution (trapezoid over the Lorentz factor, 16 Gauss nodes in pitch)."""
    e, me, cc = 4.80320471257e-10, 9.1093837015e-28, 2.99792458e10
    lx, lF, lG = table
    if thermal:
        u = torch.linspace(0.0, 1.0, 192, dtype=torch.float64, device="cuda")
        top = torch.clamp(1.0 + 45.0 * te, min=10.0) - 1.0
        gam = 1.0 + 10.0 ** (-5.0 + u[None, :] * (torch.log10(top) + 5.0)[:, None])
        f = gam * gam * torch.sqrt(torch.clamp(1.0 - 1.0 / (gam * gam), min=0.0)) * torch.exp(-gam / te[:, None])
    else:
        gam = torch.as_tensor(np.geomspace(10.0, 1.0e5, 224), device="cuda")[None, :].expand(te.numel(), -1)
        f = gam ** -3.5
    f = f / torch.trapezoid(f, gam, dim=1)[:, None]
    nu_b = e * b / (2.0 * math.pi * me * cc)
    base = torch.log(nu / (1.5 * gam * gam * nu_b[:, None]))
    mu, w = np.polynomial.legendre.leggauss(16)
    tot = [0.0, 0.0]
    for m, wt in zip(mu, w):
        sin = math.sqrt(1.0 - m * m)
        x = (base - math.log(sin)).clamp(lx[0], lx[-1])
        j = (torch.searchsorted(lx, x.contiguous(), right=True) - 1).clamp(0, 254)
        pref = 0.5 * wt * math.sqrt(3.0) * e ** 3 * sin / (me * cc ** 2)
        for q, lv in enumerate((lF, lG)):
            v = torch.exp(lv[j] + (lv[j + 1] - lv[j]) / (lx[j + 1] - lx[j]) * (x - lx[j]))
            tot[q] = tot[q] + pref * b * torch.trapezoid(f * v, gam, dim=1)
    return [n_e * t / (4.0 * math.pi) for t in tot]


def _exact_coefficients(n_e, te, b, cos, chi, nu, model):
    e, me, cc, kb, h = 4.80320471257e-10, 9.1093837015e-28, 2.99792458e10, 1.380649e-16, 6.62607015e-27
    k3, k4 = e ** 3 / (math.pi * me ** 2 * cc ** 2), e ** 4 / (4.0 * math.pi ** 2 * me ** 3 * cc ** 3)
    table = _kernel_table()
    perp, par = b * torch.sqrt(torch.clamp(1.0 - cos * cos, min=0.0)), b * cos
    out = torch.zeros((n_e.numel(), 11), dtype=torch.float64, device="cuda")

    def add(ji, jq, ai, aq, rv, rq):
        co, si = torch.cos(2.0 * chi), torch.sin(2.0 * chi)
        for k, v in zip(range(11), (ji, jq * co, jq * si, 0.0, ai, aq * co, aq * si, 0.0, rv, rq * co, rq * si)):
            out[:, k] += v

    if model in ("hybrid", "thermal"):
        ji, jq = _exact_component(n_e, te, b, nu, True, table)
        t = te * me * cc * cc / kb
        x = h * nu / (kb * t)
        planck = torch.where(x < 1e-3, 2.0 * nu * nu * kb * t / cc ** 2, 2.0 * h * nu ** 3 / cc ** 2 / torch.expm1(x))
        add(ji, jq, ji / planck, jq / planck, k3 * n_e * par / nu ** 2 * torch.clamp(1.0 / (te * te + 1.0), min=1e-8),
            k4 * n_e * perp ** 2 / nu ** 3 * te)
    if model in ("hybrid", "powerlaw"):
        n_s = 0.02 * n_e
        ji, jq = _exact_component(n_s, te, b, nu, False, table)
        g = torch.clamp(torch.sqrt(torch.clamp(nu / (4.2e6 * perp), min=1.0)), min=10.0)
        ai = ji / (g * me * nu * nu)
        pol = min(4.5 / (3.5 + 7.0 / 3.0), 0.85)
        add(ji, torch.minimum(jq, pol * ji), ai, pol * ai, 0.15 * k3 * n_s * par / nu ** 2 / 100.0,
            0.15 * k4 * n_s * perp ** 2 / nu ** 3 * math.log(1e4))
    return out


def exact(case, seed):
    """The whole images have none: a ray that grazes the spin axis, the photon orbit or the horizon amplifies the last
    bit of its state without bound, and their step-by-step loops in torch take minutes.  The network's training rounds
    its weights and activations to bfloat16 by definition."""
    kind = case["kind"]
    if kind == "points":
        grids, coeffs, pts, ini = _points_inputs(case, seed)
        parts = []
        for a in range(0, case["points"], 1 << 20):
            c, inside = _exact_samples(grids, coeffs, pts[a:a + (1 << 20)])
            if case["op"] == "step":
                s = ini.expand(c.shape[0], 4)
                c, s0 = _exact_rk2(c, 0.05, s), s
                if case["policy"] != "nan":
                    c = torch.where(inside[:, None], c, s0 if case["policy"] == "initial" else torch.zeros_like(s0))
            parts.append(c.reshape(-1))
        out = torch.cat(parts)
        return out.cpu().numpy() if case["host"] else out
    if kind == "cells":
        c, ds, ini = _cells_inputs(case, seed)
        c = c.view(-1, 11)
        s = ini.view(-1, 4).expand(c.shape[0], 4)
        if case["op"] == "rk2":
            return _exact_rk2(c, ds, s).reshape(-1)
        parts = []
        for a in range(0, c.shape[0], 1 << 18):
            k = _matrix(c[a:a + (1 << 18)])
            m = torch.zeros((k.shape[0], 5, 5), dtype=torch.float64, device="cuda")
            m[:, :4, :4] = -k * ds
            m[:, :4, 4] = c[a:a + (1 << 18), :4] * ds
            x = torch.linalg.matrix_exp(m)
            parts.append(torch.einsum("nij,nj->ni", x[:, :4, :4], s[a:a + (1 << 18)]) + x[:, :4, 4])
        return torch.cat(parts).reshape(-1)
    if kind == "frames":
        f = _frames_inputs(case, seed)
        return torch.cat([_exact_coefficients(*p.unbind(1), case["ghz"] * 1e9, case["model"])
                          for p in f.split(1 << 16)])
    if kind == "bake":
        s = _snapshot(case, seed, 0.9375)
        dev = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
        b = dev(s.b_con).view(-1, 4)
        code = torch.sqrt(b[:, 1] ** 2 + b[:, 2] ** 2 + b[:, 3] ** 2)
        n_e = dev(s.rho).view(-1) * SCALING["rho_cgs_per_code"] / 1.67262192369e-24
        cols = (n_e, dev(s.theta_e).view(-1), code * SCALING["b_gauss_per_code"], torch.zeros_like(code),
                torch.atan2(b[:, 3], b[:, 2]))
        parts = [_exact_coefficients(*(v[a:a + (1 << 17)] for v in cols), case["ghz"] * 1e9, "hybrid")
                 for a in range(0, n_e.numel(), 1 << 17)]
        return torch.cat(parts).view(s.rho.shape + (11,)).cpu().numpy()
    return None
