"""PreSCRIMP's query rows on the matrix instruction, at sizes around its blocks (8 x 8),
warps (64 windows), CTAs (32 queries x 256 windows), stages (32 elements) and the
elements it takes at once (4).  A small C++ restatement forms each cell as a chain of
fused multiply-adds in element order, which is what the instruction does: squared
distances agree bit for bit, and a differing neighbour ties."""
from __future__ import annotations

import subprocess

import numpy as np
import pytest

from thesiscode_b200 import workloads

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
typedef long long ll;
static std::vector<double> x, mu, sg, best;
static std::vector<ll> nb;
static double mm;
static double dist(double qt, ll j, ll i) { return 2.0 * (mm - (qt - mm * mu[j] * mu[i]) / (sg[j] * sg[i])); }
static void lower(ll w, double d, ll j) {
    if (d < best[w] || (d == best[w] && j < nb[w])) { best[w] = d; nb[w] = j; }
}
int main(int c, char** v) {
    const ll n = atoll(v[2]), m = atoll(v[3]), s = atoll(v[4]), PL = n - m + 1, ex = m / 4;
    x.resize(n); mu.resize(PL); sg.resize(PL); best.assign(PL, INFINITY); nb.assign(PL, 0);
    FILE* f = fopen(v[1], "rb");
    if (fread(x.data(), 8, n, f) != (size_t)n) return 2;
    mm = (double)m;
    std::vector<double> a(n), b(n);
    for (ll i = 0; i < n; ++i) { a[i] = i ? x[i] + a[i - 1] : x[i]; b[i] = i ? x[i] * x[i] + b[i - 1] : x[i] * x[i]; }
    for (ll i = 0; i < PL; ++i) {
        const double p = i ? a[m - 1 + i] - a[i - 1] : a[m - 1], q = i ? b[m - 1 + i] - b[i - 1] : b[m - 1];
        mu[i] = p / mm;
        sg[i] = std::sqrt(q / mm - mu[i] * mu[i]);
    }
    for (ll i = 0; i < PL; i += s) {
        double r = INFINITY;
        ll rj = -1;
        for (ll j = 0; j < PL; ++j) {
            if (j > i - ex && j < i + ex) continue;
            double q = 0.0;
            for (ll k = 0; k < m; ++k) q = std::fma(x[i + k], x[j + k], q);
            const double d = dist(q, j, i);
            if (d < 1.7976931348623157e308) lower(j, d, i);
            if (d < r) { r = d; rj = j; }
        }
        if (rj < 0) continue;
        lower(i, r, rj);
        const double z0 = (mm - r / 2.0) * (sg[rj] * sg[i]) + mm * mu[rj] * mu[i];
        double z = z0;
        for (ll k = 1; k < s && i + k < PL && rj + k < PL; ++k) {
            z = z - x[i + k - 1] * x[rj + k - 1] + x[i + k + m - 1] * x[rj + k + m - 1];
            const double d = dist(z, rj + k, i + k);
            if (d < 1.7976931348623157e308) { lower(i + k, d, rj + k); lower(rj + k, d, i + k); }
        }
        z = z0;
        for (ll k = 1; k < s && i - k >= 0 && rj - k >= 0; ++k) {
            z = z - x[i - k + m] * x[rj - k + m] + x[i - k] * x[rj - k];
            const double d = dist(z, rj - k, i - k);
            if (d < 1.7976931348623157e308) { lower(i - k, d, rj - k); lower(rj - k, d, i - k); }
        }
    }
    fwrite(best.data(), 8, PL, stdout);
    fwrite(nb.data(), 8, PL, stdout);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    src, exe = d / "rows.cpp", d / "rows"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-mfma", str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("kind", ["walk", "nan"])
@pytest.mark.parametrize("pl,m,step", [
    (1, 8, 3), (8, 9, 1), (9, 10, 2), (63, 11, 2), (65, 12, 9), (255, 31, 8), (257, 32, 8), (256, 33, 8),
    (511, 34, 16), (513, 35, 17), (1025, 64, 32), (2049, 67, 63), (4000, 4, 1)])
def test_rows_equal_fused_chains(gpu_ctx, program, tmp_path, kind, pl, m, step):
    n = pl + m - 1
    x = workloads.random_walk(n, pl * m)
    if kind == "nan":  # reaches the windows that hold it, and no others
        x[n // 2] = np.nan
        x[n // 4] = np.inf
    f = tmp_path / "x.bin"
    x.tofile(f)
    out = subprocess.run([program, str(f), str(n), str(m), str(step)], capture_output=True, check=True).stdout
    d2, idx = np.frombuffer(out[:8 * pl]), np.frombuffer(out[8 * pl:], dtype=np.int64)
    got = gpu_ctx.prescrimp(x, m, (step + 0.5) / m)
    assert np.array_equal(got.dist2, d2, equal_nan=True)
    for w in np.nonzero(got.index != idx)[0]:  # the keys keep the smaller of near ties
        j = int(got.index[w])
        a, b = (x[p:p + m] for p in (int(w), j))
        c = np.corrcoef(a, b)[0, 1]
        assert abs(2 * m * (1 - c) - d2[w]) <= 1e-9 * max(d2[w], 1.0), (w, j, idx[w])
