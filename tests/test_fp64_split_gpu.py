"""FP64 join with its bands cut into tiles: the same bits as the oracle's, and the
same neighbours as whole bands.  A context whose budget holds exactly what
mp_selfjoin_scratch_bytes asks for has no room for the tiles' buffers and joins
whole bands."""
from __future__ import annotations

import numpy as np
import pytest

import thesiscode_b200 as mp
from thesiscode_b200 import workloads
from tests.test_parity_gpu import check_fp64_indices

pytestmark = pytest.mark.gpu


def series(kind, n):
    rng = np.random.default_rng(n)
    if kind == "walk":
        return workloads.random_walk(n, n)
    if kind == "digital":  # small integers: many exact and near ties
        return rng.integers(0, 3, n).astype(np.float64)
    x = workloads.random_walk(n, n)  # constant stretches, NaN scores beside valid ones
    for s in range(0, n, 300):
        x[s:s + 40] = 0.0 if s % 600 else x[s]
    return x


# Columns of the longest diagonal around one and two tiles (of at least 32), around a
# band and a tile of seeds; diagonals around the band widths 32, 64, 128, 256 per
# warp; the last size walks several diagonals per thread for the tiles' first columns.
@pytest.mark.parametrize("kind", ["walk", "digital", "flat"])
@pytest.mark.parametrize("cols", [32, 33, 64, 65, 127, 129, 511, 513, 2047, 2300, 9001, 40100])
def test_tiles_equal_oracle_and_whole_bands(gpu_ctx, oracle, kind, cols):
    m = 16
    n = cols + m // 4 + 1 + m - 1
    x = series(kind, n)
    p = gpu_ctx.selfjoin(x, m, blocklen=77)
    budget = mp.load_library().mp_selfjoin_scratch_bytes(n, m, mp.FP64)
    with mp.Context(0, mem_budget_bytes=budget) as whole:
        q = whole.selfjoin(x, m, blocklen=77)
    assert np.array_equal(p.dist2, q.dist2) and np.array_equal(p.index, q.index)
    d2, idx = oracle.selfjoin(x, m, blocklen=77)
    assert np.array_equal(p.dist2, d2)
    check_fp64_indices(oracle, x, m, p.dist2, p.index, idx, blocklen=77)


@pytest.mark.parametrize("blocklen,diag", [(1, 5), (100, 40), (500, 3000), (777, 17)])
def test_block_in_tiles_equals_whole_bands(gpu_ctx, blocklen, diag):
    m = 32
    x = series("walk", 12000)
    mu, si = gpu_ctx.window_stats(x, m)
    q = gpu_ctx.first_qt(x, m, diag, diag + blocklen)
    pl = x.size - m + 1
    t = pl - diag
    xp = np.append(x, 0.0)
    got = []
    # 64-bit words per column: records 2 x 4 and their padding, keys, thresholds,
    # profile views, statistics and series -- less than the tiles' buffers add
    with mp.Context(0, mem_budget_bytes=8 * (40 * (t + 1500) + 4 * blocklen)) as whole:
        for ctx in (gpu_ctx, whole):
            prof, idx, tq = np.full(pl, -1.0), np.zeros(pl, dtype=np.int64), q.copy()
            ctx.eval_diag_block_triangle(prof[:t], idx[:t], prof[diag:], idx[diag:], tq, blocklen,
                                         t, xp, xp[diag:], m, si, mu, si[diag:], mu[diag:], diag, 0)
            got.append((prof, idx, tq))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


# The series' prefix sums run beside the tiles' first columns, in chunks of 192 values,
# 16 ahead; the first chunk starts at its second round.
@pytest.mark.parametrize("n", [191, 192, 193, 207, 208, 209, 383, 384, 385, 400, 577])
def test_prefix_sums_beside_the_tiles_equal_oracle(gpu_ctx, oracle, n):
    x, m = series("walk", n) + 40.0, 8
    p = gpu_ctx.selfjoin(x, m)
    d2, idx = oracle.selfjoin(x, m)
    assert np.array_equal(p.dist2, d2)
    check_fp64_indices(oracle, x, m, p.dist2, p.index, idx)
