"""Window statistics of the FP32 forms: the blocks that share a stretch of the series
in shared memory leave the same bits as one thread per chunk reading global memory
(division and square root by the compiler's own), which very long windows still use."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from thesiscode_b200 import build, workloads

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
int main(int argc, char** argv) {
    const int64_t n = atoll(argv[2]), m = atoll(argv[3]), PL = n - m + 1, pad = 576;
    std::vector<double> x(n), got[2], want[2];
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(x.data(), 8, n, f) != (size_t)n) return 2;
    double *A, *mean, *norm;
    int *chg, *tot;
    const int64_t blk = (n + 255) / 256;
    cudaMalloc(&A, 8 * (n + pad)); cudaMalloc(&mean, 8 * (PL + pad)); cudaMalloc(&norm, 8 * (PL + pad));
    cudaMalloc(&chg, 4 * n); cudaMalloc(&tot, 4 * (blk + 1));
    cudaMemset(A, 0xff, 8 * (n + pad)); cudaMemset(mean, 0xff, 8 * (PL + pad)); cudaMemset(norm, 0xff, 8 * (PL + pad));
    cudaMemcpy(A, x.data(), 8 * n, cudaMemcpyHostToDevice);
    launch_fp32_stats(A, m, PL, pad, chg, tot, mean, norm, 0);
    for (int k = 0; k < 2; ++k) {
        got[k].resize(PL + pad);
        want[k].assign(PL + pad, 0.0);
        cudaMemcpy(got[k].data(), k ? norm : mean, 8 * (PL + pad), cudaMemcpyDeviceToHost);
    }
    std::vector<double> tail(pad);
    cudaMemcpy(tail.data(), A + n, 8 * pad, cudaMemcpyDeviceToHost);
    for (double v : tail)
        if (v != 0.0) return 4;
    change_flags_kernel<<<grid_for(n), 256>>>(A, n, chg);
    scan_blocks_kernel<<<(unsigned)blk, 256>>>(chg, n, tot);
    scan_totals_kernel<<<1, 1>>>(tot, blk);
    scan_add_kernel<<<(unsigned)blk, 256>>>(chg, n, tot);
    welford_kernel<<<grid_for((PL + 255) / 256), 256>>>(A, m, PL, 256, chg, mean, norm);
    for (int k = 0; k < 2; ++k)
        if (cudaMemcpy(want[k].data(), k ? norm : mean, 8 * PL, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    long bad = 0, flat = 0;
    for (int k = 0; k < 2; ++k)
        for (int64_t i = 0; i < PL + pad; ++i) {
            const bool nan = got[k][i] != got[k][i] && want[k][i] != want[k][i];
            bad += !nan && memcmp(&got[k][i], &want[k][i], 8) != 0;
            flat += k == 1 && nan;
        }
    printf("windows %ld flat %ld differ %ld\n", (long)PL, flat, bad);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("stats")
    src, exe = d / "stats.cu", d / "stats"
    src.write_text(PROGRAM)
    obj = os.path.join(build.BUILD, "mp_prep.o")
    if not os.path.exists(obj):
        obj = os.path.join(build.CSRC, "mp_prep.cu")
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), obj, "-o", str(exe)], check=True)
    return str(exe)


# profiles around a chunk (256 windows), a batch (32) and a block (8,192); windows
# around 32 and 256 samples, and on both sides of the longest that a block takes
@pytest.mark.parametrize("kind", ["walk", "level", "flats", "tiny", "special"])
@pytest.mark.parametrize("pl,m", [
    (1, 2), (31, 3), (33, 31), (255, 32), (256, 33), (257, 255), (8191, 256), (8192, 257), (8193, 100),
    (20000, 1024), (9000, 8192), (300, 8193)])
def test_blocks_equal_chunks(program, tmp_path, kind, pl, m):
    n = pl + m - 1
    x = workloads.random_walk(n, n)
    if kind == "level":
        x = x * 1e-3 + 1e6
    elif kind == "flats":
        for s in range(n // 3, n, 3 * m + 50):
            x[s:s + 2 * m] = x[s] if s % 2 else 0.0
    elif kind == "tiny":  # differences outside the exponents of the short division
        x = x * 1e-290
        x[: n // 2] = np.round(x[: n // 2] * 1e290) * 1e280
    elif kind == "special":
        x[n // 2] = np.inf
        x[n // 4] = np.nan
    f = tmp_path / "x.bin"
    x.tofile(f)
    r = subprocess.run([program, str(f), str(n), str(m)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
