"""The guarded form's FP64 pass by itself: every tile is marked as touching a hazard
window, and the keys that the pass leaves are compared with direct long double
distances of every pair.  A small program built from the kernels' sources runs it."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from thesiscode_b200 import build, workloads

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
int main(int argc, char** argv) {
    const int64_t n = atoll(argv[2]), m = atoll(argv[3]), K = atoll(argv[4]), lo = atoll(argv[5]),
                  PL = n - m + 1, hi = atoll(argv[6]) < PL ? atoll(argv[6]) : PL, pad = 576;
    std::vector<double> x(n), mu(PL), nn(PL);
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(x.data(), 8, n, f) != (size_t)n) return 2;
    std::vector<int> hz(PL + 1);
    for (int64_t i = 0; i <= PL; ++i) hz[i] = (int)i;
    double *A, *mean, *norm, *df, *dg;
    int *chg, *tot, *hazard;
    unsigned long long *key, *counter;
    Fp32TileParams* desc;
    const int64_t blk = (n + 255) / 256;
    cudaMalloc(&A, 8 * (n + pad)); cudaMalloc(&mean, 8 * (PL + pad)); cudaMalloc(&norm, 8 * (PL + pad));
    cudaMalloc(&df, 8 * PL); cudaMalloc(&dg, 8 * PL); cudaMalloc(&hazard, 4 * (PL + 1));
    cudaMalloc(&chg, 4 * n); cudaMalloc(&tot, 4 * (blk + 1)); cudaMalloc(&key, 8 * PL);
    cudaMalloc(&counter, 8); cudaMalloc(&desc, sizeof(Fp32TileParams));
    cudaMemset(A, 0, 8 * (n + pad)); cudaMemset(mean, 0, 8 * (PL + pad)); cudaMemset(norm, 0, 8 * (PL + pad));
    cudaMemset(counter, 0, 8);
    cudaMemcpy(A, x.data(), 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(hazard, hz.data(), 4 * (PL + 1), cudaMemcpyHostToDevice);
    launch_fp32_stats(A, m, PL, pad, chg, tot, mean, norm, 0);
    guard_terms_kernel<<<grid_for(PL), 256>>>(A, m, PL, mean, df, dg);
    const float ulim = (float)(1.0 + 1.0 / (double)m);
    init_keys_kernel<<<grid_for(PL), 256>>>(key, PL, (unsigned long long)host_ord_f32(ulim) << 32);
    Fp32TileParams P{};
    P.A = A; P.mean = mean; P.norm = norm; P.df = df; P.dg = dg; P.hazard = hazard;
    P.m = m; P.PL = PL; P.g_lo = lo; P.g_hi = hi; P.K = reanchor_interval(K, 8); P.key = key;
    int64_t nt = 0;
    fp32_tile_plan(PL, lo, hi, P.K, 8, P.nbands, P.seg_per_pair, nt);
    cudaMemcpy(desc, &P, sizeof P, cudaMemcpyHostToDevice);
    launch_fp64_guard<8>(desc, 1, nt, counter, 0);
    std::vector<unsigned long long> got(PL);
    if (cudaMemcpy(got.data(), key, 8 * PL, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    std::vector<bool> flat(PL);
    for (int64_t i = 0; i < PL; ++i) {
        long double s = 0, q = 0;
        bool same = true;
        for (int64_t k = 0; k < m; ++k) { s += x[i + k]; same &= x[i + k] == x[i]; }
        for (int64_t k = 0; k < m; ++k) q += (x[i + k] - s / m) * (x[i + k] - s / m);
        mu[i] = (double)(s / m); nn[i] = (double)(1 / sqrtl(q)); flat[i] = same;
    }
    auto u_of = [&](int64_t i, int64_t j) {
        long double c = 0;
        for (int64_t k = 0; k < m; ++k) c += (long double)(x[i + k] - mu[i]) * (x[j + k] - mu[j]);
        return (double)(1 - c * nn[i] * nn[j]);
    };
    // u is rounded to float once (2^-24 below 1, 2^-23 below 2) after an FP64
    // recurrence that is good to far less
    const double tol = 1.3e-7;
    long bad = 0;
    for (int64_t i = 0; i < PL; ++i) {
        double best = ulim;
        for (int64_t j = 0; j < PL; ++j) {
            const int64_t g = i > j ? i - j : j - i;
            if (g < lo || g >= hi || flat[i] || flat[j]) continue;
            const double u = u_of(i, j);
            best = u < best ? u : best;
        }
        const unsigned h = (unsigned)(got[i] >> 32), b = (h & 0x80000000u) ? h & 0x7fffffffu : ~h;
        float v;
        memcpy(&v, &b, 4);
        bool ok = fabs((double)v - best) <= tol;
        if (v < ulim) ok = ok && fabs(u_of(i, (int64_t)(got[i] & 0xffffffffull)) - best) <= 2 * tol;
        bad += !ok;
    }
    printf("windows %ld off %ld\n", (long)PL, bad);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("guard")
    src, exe = d / "guard.cu", d / "guard"
    src.write_text(PROGRAM)
    objs = [os.path.join(build.BUILD, f)
            for f in ("mp_guard.o", "mp_join_fp32.o", "mp_prep.o", "mp_finalize.o")]
    if not all(os.path.exists(o) for o in objs):
        objs = [os.path.join(build.CSRC, os.path.basename(o).replace(".o", ".cu")) for o in objs]
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), *objs, "-o", str(exe)], check=True)
    return str(exe)


# around a pass (16 columns), a band (256 diagonals) and a tile; a ragged diagonal
# range; constant stretches
@pytest.mark.parametrize("flats", [False, True])
@pytest.mark.parametrize("n,m,k,lo,hi", [
    (48, 16, 64, 5, 1 << 30), (300, 16, 64, 5, 1 << 30), (545, 16, 72, 5, 1 << 30),
    (1500, 33, 1024, 9, 1 << 30), (1500, 40, 128, 100, 777)])
def test_fp64_tiles_against_direct_distances(program, tmp_path, n, m, k, lo, hi, flats):
    x = workloads.random_walk(n, n)
    if flats:
        for s in range(n // 5, n, 400):
            x[s:s + m + 6] = x[s]
    f = tmp_path / "x.bin"
    x.tofile(f)
    r = subprocess.run([program, str(f), str(n), str(m), str(k), str(lo), str(hi)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
