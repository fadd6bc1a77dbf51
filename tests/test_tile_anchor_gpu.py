"""Anchors of the FP32 form's tiles on the matrix instruction: each is the chain of
fused multiply-adds over the window in element order, bit for bit, with infinities and
NaN reaching only the windows that hold them."""
from __future__ import annotations

import subprocess

import numpy as np
import pytest

from thesiscode_b200 import build, workloads

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_tile.cuh"
using namespace mpgpu;
__global__ void anchors(Fp32TileParams P, int64_t step, double* out) {
    extern __shared__ __align__(128) char smem[];
    double nc[kTileR];
    const int64_t j0 = blockIdx.x * step, gb = P.g_lo;
    tile_anchor(P, j0, gb, gb + threadIdx.x * kTileR, threadIdx.x, smem, nc);
    for (int a = 0; a < kTileR; ++a) out[blockIdx.x * 256 + threadIdx.x * kTileR + a] = nc[a];
}
int main(int argc, char** argv) {
    const int64_t n = atoll(argv[2]), m = atoll(argv[3]), PL = n - m + 1, pad = 576, lo = 5;
    std::vector<double> x(n + pad, 0.0), mu(PL + pad, 0.0);
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(x.data(), 8, n, f) != (size_t)n) return 2;
    for (int64_t i = 0; i < PL; ++i) mu[i] = 0.25 * (double)(i % 17) - 1.0;
    const int64_t tiles = PL < 9 ? 1 : 9, step = PL < 9 ? 1 : (PL - 1) / 8;
    double *A, *mean, *out;
    cudaMalloc(&A, 8 * (n + pad)); cudaMalloc(&mean, 8 * (PL + pad)); cudaMalloc(&out, 8 * 256 * tiles);
    cudaMemcpy(A, x.data(), 8 * (n + pad), cudaMemcpyHostToDevice);
    cudaMemcpy(mean, mu.data(), 8 * (PL + pad), cudaMemcpyHostToDevice);
    Fp32TileParams P{};
    P.A = A; P.mean = mean; P.m = m; P.PL = PL; P.g_lo = lo;
    anchors<<<(unsigned)tiles, 32, kAnchorBytes>>>(P, step, out);
    std::vector<double> got(256 * tiles);
    if (cudaMemcpy(got.data(), out, 8 * got.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    long bad = 0, cells = 0;
    for (int64_t t = 0; t < tiles; ++t)
        for (int64_t d = 0; d < 256; ++d) {
            const int64_t j = t * step, r = j + lo + d;
            if (r >= PL) continue;
            double q = 0.0;
            for (int64_t k = 0; k < m; ++k) q = std::fma(x[j + k], x[r + k], q);
            const double want = std::fma((double)m * mu[j], mu[r], -q), v = got[t * 256 + d];
            bad += !(want != want && v != v) && memcmp(&want, &v, 8) != 0;
            ++cells;
        }
    printf("cells %ld differ %ld\n", cells, bad);
    return bad || (PL > 6 && !cells) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("anchor")
    src, exe = d / "anchor.cu", d / "anchor"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-Xcompiler", "-mfma,-ffp-contract=off", str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


# windows around the terms taken at once (4), a diagonal block (8) and a stage (128,
# less the 7 terms that the diagonals of a block share)
@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("pl,m", [(6, 2), (9, 3), (40, 5), (300, 8), (300, 121), (301, 122), (1000, 128),
                                  (1000, 129), (2000, 255), (700, 1000)])
def test_anchor_is_the_fused_chain(program, tmp_path, pl, m, special):
    n = pl + m - 1
    x = workloads.random_walk(n, n)
    if special:
        x[n // 2], x[n // 3] = np.inf, np.nan
    f = tmp_path / "x.bin"
    x.tofile(f)
    r = subprocess.run([program, str(f), str(n), str(m)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
