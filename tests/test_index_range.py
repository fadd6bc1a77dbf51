"""Index arithmetic of the tile kernels beyond 32-bit counts (host programs against the
kernels' headers; sizes that no test could run)."""
from __future__ import annotations

import subprocess

from thesiscode_b200 import build

HEAD = r"""
#include <cstdint>
#include <cstdio>
#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_tile.cuh"
using namespace mpgpu;
"""

# An anchor's 32-bit term count is the window's, or 0 (the plain way, which counts in 64
# bits), and the stages' positions past it stay in range.
ANCHOR = HEAD + r"""
int main() {
    int bad = 0;
    const long long e = 1ll << 31;
    for (const long long m : {2ll, 1000ll, e / 2 - 1, e / 2, e - 264, e - 8, e - 7, e, e + 5, 2 * e, 2 * e + 9, 1ll << 40}) {
        const int64_t terms = anchor_terms(m);
        const bool ok = terms == 0 ? m > 100000000 : terms == m + 7 && terms + 3 * kAnchorStep < e;
        if (!ok) std::printf("m %lld: %lld terms\n", m, (long long)terms);
        bad += !ok;
    }
    return bad;
}
"""

# Records a re-anchor interval of 2^28 columns or more away, from a tile's first.
RECORD = HEAD + r"""
int main() {
    int bad = 0;
    const long long far = 1ll << 28;
    for (const long long c : {0ll, 1000ll, far - 16, far, far + 304, 4 * far, 8 * far - 32}) {
        const int jr = (int)c;  // the tile's column count is a 32-bit one
        const uintptr_t base = 1ull << 40;
        const uintptr_t got = (uintptr_t)fp32_record((const float*)base, jr + 16);
        bad += got - base != (uintptr_t)(32 * (c + 16));
    }
    return bad;
}
"""

# PreSCRIMP's exclusion zone beside the largest window numbers: the reference's rule.
ZONE = HEAD + r"""
int main() {
    int bad = 0;
    const long long last = (1ll << 31) - 2;
    for (const long long excl : {0ll, 1ll, 16ll, 250ll, 1ll << 30, last})
        for (const long long i : {0ll, 1ll, 300ll, last / 2, last - 300, last - 1, last})
            for (const long long d : {0ll, 1ll, 15ll, 16ll, 17ll, 249ll, 250ll, 251ll, 1ll << 30, last})
                for (int s = -1; s <= 1; s += 2) {
                    const long long j = i + s * d;
                    if (j < 0 || j > last) continue;
                    const bool want = j > i - excl && j < i + excl;
                    bad += prescrimp_excluded((unsigned)i, (unsigned)j, (unsigned)excl) != want;
                }
    return bad;
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "index.cu", tmp_path / "index"
    src.write_text(program)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_anchor_of_a_window_beyond_32_bits(tmp_path):
    run(tmp_path, ANCHOR)


def test_records_beyond_32_bit_offsets(tmp_path):
    run(tmp_path, RECORD)


def test_prescrimp_exclusion_zone_of_the_last_windows(tmp_path):
    run(tmp_path, ZONE)
