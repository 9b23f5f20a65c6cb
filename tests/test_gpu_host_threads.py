"""Calls from several host threads (the C ABI's own, as a native host makes
them): each thread, on its own stream, launches one kernel with another amount
of dynamic shared memory, all above the 48 KB that need no permission.  Every
call succeeds and every result is the single-threaded one."""

from __future__ import annotations

import ctypes
import math
import shutil
import subprocess

import numpy as np
import pytest
import torch

import blackhole_native as bn
from blackhole_native import _device as dev
from blackhole_native import _lib
from blackhole_native.render import RenderConfig, Renderer

pytestmark = pytest.mark.gpu

# Every argument of the entry points called here is an integer or a pointer, which the x86-64 calling convention
# passes as 64-bit words; words past a function's own arguments are not read.
HAMMER = r"""
#include <atomic>
#include <cstdint>
#include <thread>
#include <vector>
using W = uint64_t;
using Entry = int (*)(W, W, W, W, W, W, W, W, W, W, W, W, W);
extern "C" long hammer(Entry f, const W *args, int jobs, long calls) {
    std::atomic<long> failed{0};
    std::atomic<int> ready{0};
    std::vector<std::thread> threads;
    for (int j = 0; j < jobs; ++j)
        threads.emplace_back([&, j] {
            const W *a = args + 13 * j;
            ++ready;
            while (ready.load() < jobs) std::this_thread::yield();
            for (long i = 0; i < calls; ++i)
                failed += f(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12]) != 0;
        });
    for (auto &t : threads) t.join();
    return failed;
}
"""


@pytest.fixture(scope="module")
def hammer(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler for the calling threads")
    d = tmp_path_factory.mktemp("hammer")
    (d / "h.cpp").write_text(HAMMER)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-pthread", str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    so = ctypes.CDLL(str(d / "h.so"))
    so.hammer.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint64), ctypes.c_int, ctypes.c_long]
    so.hammer.restype = ctypes.c_long

    def run(entry, jobs, calls):
        words = [w for job in jobs for w in job + [0] * (13 - len(job))]
        failed = so.hammer(ctypes.cast(entry, ctypes.c_void_p), (ctypes.c_uint64 * len(words))(*words), len(jobs), calls)
        torch.cuda.synchronize()
        return failed

    return run


def _sampler(nr, nt, np_, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(generator=g, device="cuda", dtype=torch.float64)
    keep = [torch.rand(nr * nt * np_ * 11, **f64)]
    keep += [torch.from_numpy(a).cuda() for a in (np.geomspace(1.5, 60.0, nr), np.linspace(0.05, 3.1, nt),
                                                 np.linspace(0.0, 2 * math.pi, np_, endpoint=False))]
    keep.append(torch.rand((n, 3), **f64) * torch.tensor([60.0, 3.1, 6.3], device="cuda", dtype=torch.float64) + 1.0)
    out = torch.empty(n * 11, dtype=torch.float64, device="cuda")
    c, r, t, p, pts = (dev.ptr(x) for x in keep)
    return [c, r, nr, t, nt, p, np_, pts, n, dev.ptr(out)], out, keep


def test_samplers_of_different_sizes(hammer):
    """About 51, 50, 59 and 124 KB a block: small sets, so that the threads spend their time in the calls."""
    L = _lib.lib()
    sets = [_sampler(3900, 3, 90, 2960, 1), _sampler(16, 9, 12, 60_000, 2), _sampler(2000, 3, 90, 12_400, 3),
            _sampler(3900, 3, 90, 28_000, 4)]
    want = []
    for args, out, _ in sets:
        _lib.check(L.bhn_sample_brick_trilinear(*args, dev.stream_ptr()))
        want.append(out.clone())
        out.zero_()
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    jobs = [args + [s.cuda_stream] for (args, _, _), s in zip(sets, streams)]
    assert hammer(L.bhn_sample_brick_trilinear, jobs, 30_000) == 0
    for (_, out, _), w in zip(sets, want):
        assert torch.equal(out.view(torch.int64), w.view(torch.int64))


def test_renders_of_different_bricks(hammer):
    """Bricks whose axis tables take 60 to 150 KB of a block's shared memory."""
    cfg = RenderConfig(block_threads=64, blocks_per_sm=1)
    runs = [Renderer(bn.DeviceBrick(bn.torus_brick(nr, 4, nphi, spin_a=0.9)), [bn.View(8, 8, r_obs=30.0, max_steps=4)],
                     config=cfg) for nr, nphi in ((3700, 64), (9300, 64), (5000, 32), (7000, 32))]
    want = []
    for r in runs:
        r.launch()
        want.append(r.out.clone())
        r.out.zero_()
    streams = [torch.cuda.Stream() for _ in runs]
    torch.cuda.synchronize()
    jobs, keep = [], []
    for r, s in zip(runs, streams):
        args = r._args()
        keep.append((args, r._cfg_struct, r._rays_struct))
        words = [ctypes.addressof(a._obj) if hasattr(a, "_obj") else int(a) for a in args]
        jobs.append(words + [s.cuda_stream])
    assert hammer(_lib.lib().bhn_render_launch, jobs, 10_000) == 0
    for r, w in zip(runs, want):
        assert torch.equal(r.out.view(torch.uint8), w.view(torch.uint8))
