"""Gate of the FP64 join's passes: a cell whose score exceeds a bound passes the bound's
gate, for windows of every scale, with flat, infinite and NaN terms (a host program
against the header's functions)."""
from __future__ import annotations

import subprocess

import pytest

from thesiscode_b200 import build

PROGRAM = r"""
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "mp_kernels.h"
using namespace mpgpu;
int main(int argc, char** argv) {
    const double m = atof(argv[1]);
    const int kind = atoi(argv[2]);
    std::mt19937_64 rng(kind + 1);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const double inf = INFINITY;
    const double odd[] = {0.0, -0.0, inf, -inf, NAN, 1.0, -1.0, 1e-310, -1e-310, DBL_MAX, -DBL_MAX, 0x1p200,
                          0x1p-200, -0x1p200, 0x1.8p200, 0x1p-201, 1e300, 1e-300, 3.5, -2e7};
    const int nodd = sizeof odd / sizeof *odd;
    long fails = 0, scores = 0, gated = 0;
    for (int t = 0; t < 400000; ++t) {
        double s[2], w[2], q;
        // kind 0: offsets of up to a few deviations; 1: up to 1e9; 2: any exponents; 3: odd values
        for (int k = 0; k < 2; ++k) {
            const double e = kind == 2 ? 190.0 * (2 * U(rng) - 1) : 6.0 * (2 * U(rng) - 1);
            s[k] = std::exp2(e) / std::sqrt(m);
            w[k] = (2 * U(rng) - 1) * std::sqrt(m) * (kind == 0 ? 3.0 : std::pow(10.0, 9 * U(rng)));
            if (kind == 2) w[k] = std::exp2(190.0 * (2 * U(rng) - 1)) * (rng() & 1 ? 1 : -1);
            if (kind == 3 && rng() % 2) s[k] = odd[rng() % nodd];
            if (kind == 3 && rng() % 2) w[k] = odd[rng() % nodd];
        }
        const double want = m * (kind == 2 ? std::exp2(300 * (2 * U(rng) - 1)) : U(rng));
        q = (want + w[0] * w[1]) / s[0] / s[1];
        if (kind == 3 && rng() % 2) q = odd[rng() % nodd];
        const double score = std::fma(q, s[0] * s[1], -(w[0] * w[1]));
        const double x = std::fma(-w[0], fp64_gate_mean(s[1], w[1]), s[0] * q);
        const int value = fp64_gate_value(std::max(0, high_word(x)), s[1]);
        const int err = std::max(fp64_gate_error(s[0], w[0]), fp64_gate_error(s[1], w[1]));
        for (int k = 0; k < 6; ++k) {
            const double b = k == 0 ? std::nextafter(score, -inf) : k == 1 ? score * (1 - std::exp2(-50 * U(rng)))
                           : k == 2 ? -DBL_MAX : k == 3 ? 0.0 : score - m * std::exp2(-60 * U(rng));
            if (!(score > b)) continue;
            const int g = k < 5 ? fp64_gate(b, m) : fp64_gate_high(high_word(b), fp64_gate_high_from(m));
            const int over = value + g;
            bool open = over >= 0;
            if (err > fp64_gate_errfree(m)) open = fp64_gate_lowered(g, err, over);
            fails += !open;
            ++scores;
        }
        // and it closes: a bound well above an ordinary score
        if (kind < 2 && score > 0 && score < 0.5 * m && err <= fp64_gate_errfree(m))
            gated += value + fp64_gate(score * 1.001 + 1e-4 * m, m) < 0;
    }
    printf("scores %ld missed %ld closed %ld\n", scores, fails, gated);
    return fails || scores < 100000 || (kind == 0 && gated < 100000);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("gate")
    src, exe = d / "gate.cu", d / "gate"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-Xcompiler", "-mfma,-ffp-contract=off", str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("m", [4, 100, 1024])
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_no_cell_above_its_bound_is_missed(program, m, kind):
    r = subprocess.run([program, str(m), str(kind)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
