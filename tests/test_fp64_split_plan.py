"""Buffers of the FP64 join's tiles on CPU: the rows that two tiles of a band meet have places of
their own, and the buffers stay small beside the join's other scratch."""
from __future__ import annotations

import os
import subprocess

import thesiscode_b200 as mp
from thesiscode_b200 import build

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <vector>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
// seam rows of a tile: t < span (a tile before it) and t >= L (one after it), t < L + span
static int slots(int64_t L, int64_t span) {
    std::vector<int> taken((size_t)fp64_seam_rows(L, span), 0);
    int bad = fp64_seam_rows(L, span) > 2 * span;
    for (int64_t t = 0; t < L + span; ++t) {
        if (t >= span && t < L) continue;
        const int64_t i = fp64_seam_slot(t, L, span);
        if (i < 0 || i >= fp64_seam_rows(L, span) || taken[(size_t)i]++) ++bad;
    }
    return bad;
}
int main() {
    int bad = 0;
    for (int64_t span : {32, 64, 128, 256})
        for (int64_t L = 32; L < 1200; L += 16) bad += slots(L, span);
    for (int64_t span : {32, 256}) bad += slots(200000, span);
    const int64_t sizes[][3] = {  // columns, diagonals [lo, hi)
        {300, 5, 300}, {2401, 26, 2401}, {16129, 65, 16129}, {65137, 101, 65137}, {131000, 65, 131000},
        {199745, 65, 199745}, {242000, 65, 242000}, {45036, 0, 500}, {400000, 1000, 21000}, {8387585, 257, 33025},
        {8387585, 100000, 300000}};
    for (const auto& z : sizes)
        for (int R : {1, 2, 4, 8}) {
            const Fp64Split S = fp64_split_plan(z[0], z[1], z[2], R);
            const size_t bytes = fp64_split_bytes(S, z[2] - z[1], R);
            // 5 tiles for each of 1,184 warps and a partial one per band, 64R rows of 12 bytes each;
            // and a number per tile of each diagonal, 256 diagonals to 32 columns or more
            if (bytes > (size_t)(100 << 20)) {
                std::printf("%lld columns, R %d: %zu bytes\n", (long long)z[0], R, bytes);
                ++bad;
            }
        }
    // in the place of a join's key shards but one (16 bytes per window each, 32 MB in all)
    for (int64_t n : {600, 1000, 2500, 4000, 8000, 16384, 40000, 65536, 100000, 131072, 180000, 240000}) {
        const int64_t shards = std::max<int64_t>(1, std::min<int64_t>(16, 2000000 / n));
        const size_t room = (size_t)(16 * n * (shards - 1));
        const int R = n < 2065 ? 4 : 8;
        const Fp64Split S = fp64_split_plan(n, 17, n, R, room), T = fp64_split_plan(n, 17, n, R);
        const bool ok = S.L >= T.L && S.L % kFp64SplitUnit == 0 && S.L < n - 17 &&
                        fp64_split_bytes(S, n - 17, R) <= room && fp64_split_plan(n, 17, n, R, 1000).L == 0;
        if (!ok) std::printf("n %lld: L %lld (%lld with room)\n", (long long)n, (long long)S.L, (long long)T.L);
        bad += !ok;
    }
    return bad != 0;
}
"""


def test_seams_of_the_tiles(tmp_path):
    src, exe = tmp_path / "seams.cu", tmp_path / "seams"
    src.write_text(PROGRAM)
    libdir = os.path.dirname(mp.LIB_PATH)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), "-o", str(exe), f"-L{libdir}", "-lmpgpu",
                    "-Xlinker", f"-rpath={libdir}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
