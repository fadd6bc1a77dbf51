"""FP64 join over whole bands on data whose gates open often or whose windows have no finite
score: the oracle's bits, and those of bands cut into tiles."""
from __future__ import annotations

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
@pytest.mark.parametrize("n,m", [(2400, 8), (9001, 16), (9001, 300)])
def test_whole_bands_equal_oracle_and_tiles(gpu_ctx, oracle, kind, n, m):
    x = series(kind, n)
    budget = mp.load_library().mp_selfjoin_scratch_bytes(n, m, mp.FP64)
    with mp.Context(0, mem_budget_bytes=budget) as whole:  # no room for the tiles' buffers
        p = whole.selfjoin(x, m)
        launches = whole.last_launch_count
    q = gpu_ctx.selfjoin(x, m)
    assert launches < gpu_ctx.last_launch_count  # seeds and seams
    assert np.array_equal(p.dist2, q.dist2) and np.array_equal(p.index, q.index)
    if kind == "nan":
        return  # the oracle's statistics differ there
    d2, idx = oracle.selfjoin(x, m)
    assert np.array_equal(p.dist2, d2, equal_nan=True)
    if kind not in ("steps", "signs"):  # infinite or equal scores tie by the thousand there
        check_fp64_indices(oracle, x, m, p.dist2, p.index, idx)
