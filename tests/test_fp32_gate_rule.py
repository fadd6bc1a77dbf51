"""Rules of the FP32 forms' gates on CPU: what bound a key sets, and which joins go behind the
gate (host programs against the header's functions)."""
from __future__ import annotations

import subprocess

from thesiscode_b200 import build

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
static float value(unsigned bits) { float x; std::memcpy(&x, &bits, 4); return x; }
int main() {
    int bad = 0;
    const unsigned long long init = (unsigned long long)host_ord_f32(1.01f) << 32;
    // a window's first key: one that every distance below it replaces, or none does
    bad += fp32_first_key(init, 0.5) != init || fp32_first_key(init, INFINITY) != init;
    bad += fp32_first_key(init, NAN) != kFp32FlatKey || kFp32FlatKey < init;
    for (int tags = 0; tags < 2; ++tags) {
        bad += fp32_key_bound((unsigned)(kFp32FlatKey >> 32), tags) != 0;  // nothing concerns a flat window
        bad += !(value(fp32_key_bound((unsigned)(init >> 32), tags)) >= 1.01f);
    }
    std::mt19937 rng(3);
    std::uniform_real_distribution<float> U(-0.2f, 1.2f);
    for (int t = 0; t < 200000; ++t) {
        const float u = U(rng);
        const unsigned exact = fp32_key_bound(host_ord_f32(u), false), tagged = fp32_key_bound(host_ord_f32(u), true);
        if (u < 0.f) {
            bad += exact != 0 || tagged != 0;
            continue;
        }
        bad += value(exact) != u;
        unsigned b;
        std::memcpy(&b, &u, 4);
        bad += !(tagged > (b | 0xffu)) || tagged > (b | 0xffu) + 1;  // above all its tags, below the next value
    }
    std::printf("%d wrong\n", bad);
    return bad != 0;
}
"""

# Joins whose tiles of 1,024 columns are one wave of the selecting passes' resident warps (12
# on each of 148 SMs) select in every pass.
WAY = r"""
#include <cstdio>
#include "mp_common.cuh"
#include "mp_kernels.h"
using namespace mpgpu;
int main() {
    int bad = 0;
    for (const long long m : {170ll, 256ll, 400ll, 1024ll})
        for (long long n = 24000; n < 60000; n += 500) {
            Fp32TileParams P{};
            P.m = m;
            P.PL = n - m + 1;
            long long tiles = 0;  // with work (a pair of bands leaves some numbers unused)
            for (long long g = m / 4 + 1; g < P.PL; g += 256) tiles += (P.PL - g + 1023) / 1024;
            const Fp32Way way = fp32_way_of(&P, 1);
            if (tiles <= 148 * 12 - 60 && way != kFp32Dense) ++bad, std::printf("%lld / %lld dense\n", n, m);
            if (tiles > 148 * 12 + 120 && way != kFp32Gate) ++bad, std::printf("%lld / %lld gate\n", n, m);
        }
    return bad != 0;
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "rule.cu", tmp_path / "rule"
    src.write_text(program)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_bounds_of_keys(tmp_path):
    run(tmp_path, PROGRAM)


def test_one_wave_of_tiles_selects(tmp_path):
    run(tmp_path, WAY)
