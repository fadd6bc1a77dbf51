"""Windows without a finite score (constant ones, or with a NaN) in the FP64 join's gate: it stays
shut for their cells, except where a score is infinite (a host program against the header's
functions)."""
from __future__ import annotations

import subprocess

from thesiscode_b200 import build

PROGRAM = r"""
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <random>
#include "mp_kernels.h"
using namespace mpgpu;
int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    const double inf = INFINITY, m = 100;
    const double odd[][2] = {{NAN, NAN}, {NAN, 1.0}, {inf, NAN}, {inf, inf}, {inf, -inf}, {1.0, NAN}};
    long missed = 0, open = 0, infinite = 0, cells = 0;
    for (int t = 0; t < 300000; ++t)
        for (const auto& o : odd)
            for (int flip = 0; flip < 2; ++flip) {
                // an ordinary window, its mean term down to the smallest numbers
                const double s = std::exp2(40 * U(rng)), w = t % 8 ? 30 * U(rng) : U(rng) * std::exp2(-1000 + 300 * U(rng));
                const double q = std::exp2(50 * U(rng)) * (rng() & 1 ? 1 : -1);
                const double s0 = flip ? s : o[0], w0 = flip ? w : o[1];  // row
                const double s1 = flip ? o[0] : s, w1 = flip ? o[1] : w;  // column
                const double score = std::fma(q, s0 * s1, -(w0 * w1));
                const double x = std::fma(-w0, fp64_gate_mean(s1, w1), s0 * q);
                const int value = fp64_gate_value(std::max(0, high_word(x)), s1);
                const double start = fp64_bound(-DBL_MAX, o[0], o[1]);
                const int gate = fp64_gate(start, m), again = fp64_gate_high(high_word(start), fp64_gate_high_from(m));
                if (score > start) {
                    ++infinite;
                    missed += value + gate < 0 || value + again < 0;
                } else if (!flip) {  // (a constant column's value is infinite for any cell)
                    // a NaN's sign is the machine's own: not looked at
                    open += !std::isnan(x) && (value + gate >= 0 || value + again >= 0);
                }
                // the test of a score by itself
                const int hi = fp64_cell_high(high_word(score));
                const bool row = hi + fp64_best_gate(high_word(start)) >= kFp64Pass;
                const bool col = hi + fp64_cell_gate(gate) >= kFp64Pass;
                missed += score > start && !(row && col);
                open += !(score > start) && (row || col);
                // ... against an ordinary window's best, or none yet
                for (const double b : {-DBL_MAX, -0.5, -0.0, 0.0, 1e-300, 0.7, 99.0, score, 0.999 * score}) {
                    const bool pass = hi + fp64_best_gate(high_word(b)) >= kFp64Pass;
                    missed += score > b && !pass;
                    open += !(score > b) && b > 0.0 && (std::isnan(score) || score < 0.99 * b) && pass;
                }
                ++cells;
            }
    // an ordinary window keeps its threshold
    const bool kept = fp64_bound(3.5, 2.0, 1.0) == 3.5 && fp64_bound(-DBL_MAX, 0.0, 0.0) == -DBL_MAX;
    printf("cells %ld infinite %ld missed %ld open %ld\n", cells, infinite, missed, open);
    return missed || open || infinite < 1000 || !kept;
}
"""


def test_gate_of_windows_without_a_finite_score(tmp_path):
    src, exe = tmp_path / "bounds.cu", tmp_path / "bounds"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-Xcompiler", "-mfma,-ffp-contract=off", str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
