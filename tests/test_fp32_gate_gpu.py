"""FP32 join: the passes behind the gate, the passes that all select and the mix of
both leave the same keys, bit for bit.  A small program built from the kernels'
sources runs every way on the same records."""
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
#include <vector>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
int main(int argc, char** argv) {
    const int64_t n = atoll(argv[2]), m = atoll(argv[3]), K = atoll(argv[4]), lo = atoll(argv[5]),
                  hi = atoll(argv[6]), PL = n - m + 1, pad = 576;
    std::vector<double> x(n);
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(x.data(), 8, n, f) != (size_t)n) return 2;
    double *A, *mean, *norm;
    int *chg, *tot;
    float4 *row, *col;
    unsigned long long *key, *counter;
    Fp32TileParams* desc;
    const int64_t blk = (n + 255) / 256;
    cudaMalloc(&A, 8 * (n + pad)); cudaMalloc(&mean, 8 * (PL + pad)); cudaMalloc(&norm, 8 * (PL + pad));
    cudaMalloc(&chg, 4 * n); cudaMalloc(&tot, 4 * (blk + 1)); cudaMalloc(&row, 32 * (PL + pad));
    cudaMalloc(&col, 32 * (PL + pad)); cudaMalloc(&key, 8 * PL); cudaMalloc(&counter, 8);
    cudaMalloc(&desc, sizeof(Fp32TileParams));
    cudaMemset(A, 0, 8 * (n + pad)); cudaMemset(mean, 0, 8 * (PL + pad)); cudaMemset(norm, 0, 8 * (PL + pad));
    cudaMemcpy(A, x.data(), 8 * n, cudaMemcpyHostToDevice);
    launch_fp32_stats(A, m, PL, pad, chg, tot, mean, norm, 0);
    pack_fp32_kernel<<<grid_for(PL + pad), 256>>>(A, m, PL, 4, PL + pad, mean, norm, row, col, key, 0ull,
                                                  Fp32TileParams{}, nullptr, nullptr);
    Fp32TileParams P{};
    P.rowrec = row; P.colrec = col; P.A = A; P.mean = mean; P.m = m; P.PL = PL;
    P.g_lo = lo; P.g_hi = hi < PL ? hi : PL; P.K = reanchor_interval(K, 8); P.key = key;
    int64_t nt = 0;
    fp32_tile_plan(PL, P.g_lo, P.g_hi, P.K, 8, P.nbands, P.seg_per_pair, nt);
    cudaMemcpy(desc, &P, sizeof P, cudaMemcpyHostToDevice);
    std::vector<unsigned long long> first(PL), got(PL);
    const unsigned long long init = (unsigned long long)host_ord_f32((float)(1.0 + 1.0 / (double)m)) << 32;
    for (int group = 0; group < 2; ++group)
        for (int way = 0; way < (group ? 2 : 3); ++way) {
            init_keys_kernel<<<grid_for(PL), 256>>>(key, PL, init);
            cudaMemset(counter, 0, 8);
            launch_fp32_join<8>(desc, 1, nt, counter, 0, (Fp32Way)way, group != 0);
            auto& to = way == 0 ? first : got;
            if (cudaMemcpy(to.data(), key, 8 * PL, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
            if (way == 0) {
                long found = 0;
                for (int64_t i = 0; i < PL; ++i) found += first[i] != init;
                printf("found %ld\n", found);
                continue;
            }
            long bad = 0;
            for (int64_t i = 0; i < PL; ++i) bad += got[i] != first[i];
            printf("group %d way %d differ %ld\n", group, way, bad);
            if (bad) return 1;
        }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ways")
    src, exe = d / "ways.cu", d / "ways"
    src.write_text(PROGRAM)
    objs = [os.path.join(build.BUILD, f) for f in ("mp_join_fp32.o", "mp_prep.o", "mp_finalize.o")]
    if not all(os.path.exists(o) for o in objs):
        objs = [os.path.join(build.CSRC, os.path.basename(o).replace(".o", ".cu")) for o in objs]
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), *objs, "-o", str(exe)], check=True)
    return str(exe)


def series(kind, n):
    rng = np.random.default_rng(n)
    t = np.arange(n)
    if kind == "walk":
        return workloads.random_walk(n, n)
    if kind == "repeats":  # exact repeats: distances at and below 0 in FP32
        return np.tile(workloads.random_walk((n + 3) // 4, 1), 4)[:n]
    if kind == "flats":  # flat windows (NaN norms) and level steps
        x = workloads.random_walk(n, 3)
        for s in range(0, n, 1500):
            x[s:s + 700] = 0.0 if s % 3000 else x[s]
        return x
    if kind == "digital":
        return rng.integers(0, 3, n).astype(np.float64)
    return np.sin(2e-6 * t * t) + 0.01 * rng.standard_normal(n)  # chirp: neighbours keep improving


# window, interval and sizes around a pass (16 columns), a band (256 diagonals) and a
# tile; diagonal ranges that leave a band ragged
@pytest.mark.parametrize("kind", ["walk", "repeats", "flats", "digital", "chirp"])
@pytest.mark.parametrize("n,m,k,lo,hi", [
    (300, 16, 64, 5, 1 << 30), (1040, 16, 72, 5, 1 << 30), (5001, 64, 256, 17, 1 << 30),
    (9000, 200, 1024, 51, 3333), (30011, 100, 1024, 26, 1 << 30), (30011, 1000, 64, 251, 1 << 30),
    (120000, 250, 1000, 4000, 12347)])
def test_every_way_leaves_the_same_keys(program, tmp_path, kind, n, m, k, lo, hi):
    f = tmp_path / "x.bin"
    series(kind, n).tofile(f)
    r = subprocess.run([program, str(f), str(n), str(m), str(k), str(lo), str(hi)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    # (the shortest series with flats is one constant stretch)
    assert int(r.stdout.split()[1]) > 0 or (kind == "flats" and n <= 700)
