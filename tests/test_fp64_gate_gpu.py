"""FP64 join on series whose windows reach the ends of the gate's rule (large offsets, extreme
scales, constant stretches of either sign, one huge value): the oracle's bits."""
from __future__ import annotations

import numpy as np
import pytest

from thesiscode_b200 import workloads
from tests.test_parity_gpu import check_fp64_indices

pytestmark = pytest.mark.gpu


def series(kind, n):
    x = workloads.random_walk(n, n)
    if kind == "offset":
        return x + 3e5
    if kind == "small":
        return x * 1e-75
    if kind == "large":
        return x * 1e75
    if kind == "levels":  # constant stretches of alternating sign between ordinary windows
        for k, s in enumerate(range(0, n - 200, 450)):
            x[s:s + 150] = 7.25 if k % 2 else -7.25
        return x
    x[n // 2] = 1e9  # spike: windows with a large scale and mean term beside ordinary ones
    return x


@pytest.mark.parametrize("kind", ["offset", "small", "large", "levels", "spike"])
@pytest.mark.parametrize("n,m", [(1500, 16), (9001, 64), (20000, 100)])
def test_join_equals_oracle(gpu_ctx, oracle, kind, n, m):
    x = series(kind, n)
    p = gpu_ctx.selfjoin(x, m)
    d2, idx = oracle.selfjoin(x, m)
    assert np.array_equal(p.dist2, d2, equal_nan=True)
    if kind != "levels":  # infinite scores tie by the thousand there
        check_fp64_indices(oracle, x, m, p.dist2, p.index, idx)
