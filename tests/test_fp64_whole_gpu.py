"""FP64 join over whole bands and over tiles of any length on data whose gates open often or
whose windows have no finite score: the oracle's bits, and one another's."""
from __future__ import annotations

import re

import numpy as np
import pytest

import thesiscode_b200 as mp
from thesiscode_b200 import workloads
from tests.test_parity_gpu import check_fp64_indices

pytestmark = pytest.mark.gpu


def series(kind, n):
    rng = np.random.default_rng(n)
    if kind == "noise":
        return rng.standard_normal(n)
    if kind == "sine":  # a noisy pattern that comes again and again
        return np.sin(2 * np.pi * np.arange(n) / 97.3) + 0.1 * rng.standard_normal(n)
    if kind == "steps":  # constant windows, and exact ties among all others
        return np.repeat(rng.integers(-5, 6, n // 150 + 1), 150)[:n].astype(np.float64)
    x = workloads.random_walk(n, n)
    if kind == "nan":
        x[n // 2] = np.nan
    elif kind == "signs":  # constant windows of either sign beside ordinary ones
        for k, s in enumerate(range(0, n - 200, 450)):
            x[s:s + 150] = 7.25 if k % 2 else -7.25
    return x


@pytest.mark.parametrize("kind", ["walk", "noise", "sine", "steps", "nan", "signs"])
@pytest.mark.parametrize("n,m", [(150, 8), (700, 8), (2400, 8), (9001, 16), (9001, 300)])
def test_join_in_its_stated_scratch_equals_oracle(gpu_ctx, oracle, kind, n, m):
    x = series(kind, n)
    budget = mp.load_library().mp_selfjoin_scratch_bytes(n, m, mp.FP64)
    with mp.Context(0, mem_budget_bytes=budget) as stated:  # longer tiles in the key shards' place
        p = stated.selfjoin(x, m)
        launches = stated.last_launch_count
    q = gpu_ctx.selfjoin(x, m)
    assert launches == gpu_ctx.last_launch_count  # tiles in both: seeds and seams
    assert np.array_equal(p.dist2, q.dist2) and np.array_equal(p.index, q.index)
    if kind == "nan":
        return  # the oracle's statistics differ there
    d2, idx = oracle.selfjoin(x, m)
    assert np.array_equal(p.dist2, d2, equal_nan=True)
    if kind not in ("steps", "signs"):  # infinite or equal scores tie by the thousand there
        check_fp64_indices(oracle, x, m, p.dist2, p.index, idx)


# Above 947 bands of 256 diagonals the bands stay whole; two ranges of half the diagonals
# each are cut into tiles.
@pytest.mark.parametrize("kind", ["walk", "noise", "sine", "steps", "nan", "signs"])
@pytest.mark.parametrize("m", [8, 100])
def test_wide_whole_bands_equal_two_ranges_in_tiles(gpu_ctx, kind, m):
    n = 243000 + m
    x = series(kind, n)
    p = gpu_ctx.selfjoin(x, m)
    launches = gpu_ctx.last_launch_count
    pl, mid = n - m + 1, 100001
    q = gpu_ctx.selfjoin_ranges(x, m, [(m // 4 + 1, mid), (mid, pl)])
    assert gpu_ctx.last_launch_count >= launches + 4  # another join, seeds and seams twice
    assert np.array_equal(p.dist2, q.dist2, equal_nan=True) and np.array_equal(p.index, q.index)


def block(ctx, x, m, diag, blocklen, q, mu, si):
    pl = x.size - m + 1
    t = pl - diag
    xp = np.append(x, 0.0)
    prof, idx, tq = np.full(pl, -1.0), np.zeros(pl, dtype=np.int64), q.copy()
    ctx.eval_diag_block_triangle(prof[:t], idx[:t], prof[diag:], idx[diag:], tq, blocklen, t, xp,
                                 xp[diag:], m, si, mu, si[diag:], mu[diag:], diag, 0)
    return prof, idx, tq


# The budget that leaves no room for tiles is what the call itself says it needs.
@pytest.mark.parametrize("kind", ["walk", "steps"])
@pytest.mark.parametrize("blocklen,diag", [(1, 5), (31, 900), (100, 40), (500, 3000), (777, 17), (2100, 60)])
def test_block_in_tiles_equals_whole_bands_by_path(gpu_ctx, kind, blocklen, diag):
    m = 32
    x = series(kind, 12000)
    with np.errstate(all="ignore"):
        mu, si = gpu_ctx.window_stats(x, m)
    q = gpu_ctx.first_qt(x, m, diag, diag + blocklen)
    got = block(gpu_ctx, x, m, diag, blocklen, q, mu, si)
    launches = gpu_ctx.last_launch_count
    with mp.Context(0, mem_budget_bytes=1) as none, pytest.raises(mp.MpError) as e:
        block(none, x, m, diag, blocklen, q, mu, si)
    need = int(re.search(r"needs (\d+) bytes", str(e.value)).group(1))
    with mp.Context(0, mem_budget_bytes=need) as whole:
        want = block(whole, x, m, diag, blocklen, q, mu, si)
        assert whole.last_launch_count == launches - 2  # seeds and seams
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
