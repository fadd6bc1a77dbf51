"""What a call costs on other data than random walks, beside a walk of the same size (series
of constant stretches, with a NaN, with a short pattern that comes again and again), and
what it costs where there is no room for the fastest way."""
from __future__ import annotations

import time

import numpy as np
import pytest

import thesiscode_b200 as mp
from thesiscode_b200 import workloads

pytestmark = pytest.mark.gpu


def series(kind, n):
    x = workloads.random_walk(n, n)
    if kind == "nan":  # prefix sums: every window from its first one on is NaN
        x[n // 2] = np.nan
    elif kind == "constant":
        x[:] = 3.7
    elif kind == "sine":
        x = np.sin(2 * np.pi * np.arange(n) / 97.3) + 0.1 * np.random.default_rng(n).standard_normal(n)
    elif kind == "steps":
        x = np.repeat(np.random.default_rng(n).integers(-5, 6, n // 150 + 1), 150)[:n].astype(np.float64)
    return x


def on_gpu(x, m):
    import torch
    return torch.from_numpy(x).cuda(), (torch.empty(x.size - m + 1, dtype=torch.float64, device="cuda"),
                                        torch.empty(x.size - m + 1, dtype=torch.int64, device="cuda"))


def ms(call, runs=7):
    import torch
    best = 1e9
    for _ in range(runs):
        torch.cuda.synchronize()
        t = time.perf_counter()
        call()  # returns when the result is there
        best = min(best, time.perf_counter() - t)
    return 1e3 * best


# Walks take 5.5 ms here, and 7.0 where the rows ran without the matrix instruction; these
# series took 7.5 and 7.7 then.
@pytest.mark.parametrize("kind", ["nan", "constant"])
def test_prescrimp_of_degenerate_windows(gpu_ctx, kind):
    n, m = 100000, 64
    t = []
    for k in ("walk", kind):
        x, out = on_gpu(series(k, n), m)
        t.append(ms(lambda: gpu_ctx.prescrimp(x, m, 0.25, out=out)))
    assert t[1] < 1.35 * t[0], t


# 280,000 samples (whole bands): a walk with m = 256 takes about 28 ms; with every step tested
# in FP64 all of these took 43 ms, the steps 60.
@pytest.mark.parametrize("kind,m,limit", [("walk", 16, 1.9), ("sine", 32, 1.9), ("nan", 64, 1.9),
                                          ("steps", 256, 3.0)])
def test_fp64_join_where_gates_open(gpu_ctx, kind, m, limit):
    n = 280000
    t = []
    for k, w in (("walk", 256), (kind, m)):
        x, out = on_gpu(series(k, n), w)
        t.append(ms(lambda: gpu_ctx.selfjoin(x, w, out=out), runs=3))
    assert t[1] < limit * t[0], t


# 2,500 samples in short tiles take 0.14 ms a call, 0.96 in whole bands, on 10 warps.
def test_fp64_join_in_its_stated_scratch(gpu_ctx):
    n, m = 2500, 100
    x, out = on_gpu(series("walk", n), m)
    budget = mp.load_library().mp_selfjoin_scratch_bytes(n, m, mp.FP64)
    with mp.Context(0, mem_budget_bytes=budget) as stated:
        t = [ms(lambda: c.selfjoin(x, m, out=out), runs=30) for c in (gpu_ctx, stated)]
    assert t[1] < 4.0 * t[0], t


# A walk takes 1.7 ms a call; with a NaN, whose stretches' anchors are summed the plain way,
# 2.4 where every anchor was, and 7.1 where both ways were taken one after the other.
def test_fp32_join_with_a_nan_in_long_windows(gpu_ctx):
    n, m = 60000, 8192
    t = []
    for kind in ("walk", "nan"):
        x, out = on_gpu(series(kind, n), m)
        t.append(ms(lambda: gpu_ctx.selfjoin(x, m, precision=mp.FP32_REANCHOR, out=out)))
    assert t[1] < 3.0 * t[0], t


# The last block of the statistics walks zeros past the profile's end: 5,000 samples with
# windows of 1,200 in 0.2 ms a call, 0.55 with a division for each; a walk of 60,000 and 400
# takes 0.6.
def test_fp32_join_of_a_short_profile_with_long_windows(gpu_ctx):
    t = []
    for n, m in ((60000, 400), (5000, 1200)):
        x, out = on_gpu(series("walk", n), m)
        t.append(ms(lambda: gpu_ctx.selfjoin(x, m, precision=mp.FP32_REANCHOR, out=out), runs=15))
    assert t[1] < 0.6 * t[0], t
