// Shared by the kernels that walk the FP32 form's tiles (32 * kTileR adjacent
// diagonals by K columns, one warp each): the FP32 join and the guarded form's
// FP64 pass.
#pragma once

#include "mp_common.cuh"
#include "mp_kernels.h"

namespace mpgpu {

constexpr int kTileR = 8;  // diagonals per lane

// First dot products of a tile: q[a] = sum_k A[j0 + k] A[j0 + g0 + a + k], summed in
// k order with fused operations, for the lane's diagonals g0 + a, g0 = gb + 8 lane.
//
// On the FP64 matrix instruction: with diagonal gb + 8p + s (p < 32, s < 8) and k' = k
// + s, the products are X Y with X[s][k'] = A[j0 + k' - s] inside the window (0
// outside) and Y[k'][p] = A[j0 + gb + 8p + k'] -- 8 x 32 results, m + 7 terms each in
// k order, the zeros before and after changing nothing.  Both operands come from
// stretches of the series that the warp stages in its (not yet used) shared memory.
// Four instructions per 4 terms leave the other warps the issue slots and registers
// that 32 multiply-adds and their operands took.  n = 300,007, m = 1000, K = 256
// (3.9 products per cell): 23.5 -> 19.0 ms.
// A stretch with an infinity or NaN is summed the plain way from its first term on: 0
// times it is NaN (60,000 samples, m = 8192, a NaN in the middle: 1.4 ms a join; 4.7 with
// all stages before it and its sums kept in memory).
constexpr int kAnchorStep = 128;                       // terms k' per stage
constexpr int kAnchorY = (kAnchorStep + 256) / 8 * 12;  // element i at i + 4 (i / 8): conflict-free
constexpr int kAnchorBytes = 8 * (kAnchorStep + 8 + kAnchorY + 256);
constexpr int kAnchorChunk = 320;                      // terms per stage of the plain way
static_assert(8 * (kAnchorChunk + (32 * kTileR + kAnchorChunk) * 9 / 8) <= kAnchorBytes, "one area for both");
// Terms of a window's product, counted in 32 bits with room for a stage (64-bit counts cost
// 0.7 to 4% of a join with K = 256); 0 for a longer window, which is summed the plain way.
// (Host-callable, so the rule can be checked without a GPU.)
__host__ __device__ inline int anchor_terms(int64_t m) { return m < (int64_t(1) << 30) ? (int)m + 7 : 0; }

// The plain way, the lane's sums to out[0 .. 7] (in `area` too, once the terms have been
// read).  The series terms are staged CHUNK at a time: the column's A[j0 + k] and the
// warp's rows A[j0 + gb + i], i < 32R + chunk, skewed by one double per 8 so that lanes
// reading rows 8 apart hit distinct banks.
template <int CHUNK>
__device__ __noinline__ void tile_anchor_scalar(const double* A, int64_t m, int64_t j0, int64_t gb, int lane,
                                                char* area, double* out) {
    constexpr int R = kTileR;
    double q[R];
#pragma unroll
    for (int a = 0; a < R; ++a) q[a] = 0.0;
    {
        static_assert(R % 8 == 0, "anchor row skew assumes lanes start on multiples of 8 rows");
        double* scol = reinterpret_cast<double*>(area);
        double* srow = scol + CHUNK;
        const double* Ac = A + j0;
        const double* Ar = A + j0 + gb;
        // lane's rows i = lane*R + t sit at srow[lane*(R + R/8) + t + t/8]
        const double* wl = srow + lane * (R + R / 8);
        for (int64_t kb0 = 0; kb0 < m; kb0 += CHUNK) {
            const int kc = (int)min((int64_t)CHUNK, m - kb0);
            __syncwarp();
#pragma unroll 4
            for (int i = lane; i < kc; i += 32) scol[i] = __ldg(Ac + kb0 + i);
#pragma unroll 4
            for (int i = lane; i < 32 * R + kc; i += 32) srow[i + (i >> 3)] = __ldg(Ar + kb0 + i);
            __syncwarp();
            double w[R];
#pragma unroll
            for (int a = 0; a < R - 1; ++a) w[a] = wl[a];
            int k = 0;
            for (; k + R <= kc; k += R) {
                const double* wk = wl + (k / 8) * 9;  // row lane*R + k, k % 8 == 0
#pragma unroll
                for (int kk = 0; kk < R; ++kk) {
                    const int t = kk + R - 1;
                    w[(kk + R - 1) % R] = wk[t + (t >> 3)];
                    const double x = scol[k + kk];
#pragma unroll
                    for (int a = 0; a < R; ++a) q[a] = __fma_rn(x, w[(kk + a) % R], q[a]);
                }
            }
            for (; k < kc; ++k) {
                const double x = scol[k];
#pragma unroll
                for (int a = 0; a < R; ++a) {
                    const int t = k + a;
                    q[a] = __fma_rn(x, wl[t + (t >> 3)], q[a]);
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int a = 0; a < R; ++a) out[a] = q[a];
}

// FP64 re-anchor of a tile: minus the covariance at its first column j0 of the lane's
// diagonals, m mean_j0 mean_r - q.  area: kAnchorBytes of the warp's shared memory.
__device__ __forceinline__ void tile_anchor(const Fp32TileParams& P, int64_t j0, int64_t gb, int64_t g0,
                                            int lane, char* area, double (&nc)[kTileR]) {
    double* sx = reinterpret_cast<double*>(area);  // term k0 - 8 + i at i
    double* sy = sx + kAnchorStep + 8;
    double* sq = sy + kAnchorY;
    const int lr = lane >> 2, lc = lane & 3;
    const double* Ax = P.A + j0;
    const double* Ay = P.A + j0 + gb;
    double c[4][2];
#pragma unroll
    for (int p = 0; p < 4; ++p) c[p][0] = c[p][1] = 0.0;
    const int terms = anchor_terms(P.m);
    bool finite = terms > 0;
    // a stage's values go through registers, read while the stage before it runs
    constexpr int NX = (kAnchorStep + 8 + 31) / 32, NY = (kAnchorStep + 256) / 32;
    double rx[NX], ry[NY];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            const int k = k0 - 8 + 32 * i + lane;
            rx[i] = k >= 0 && k < (int)P.m ? __ldg(Ax + k) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < NY; ++i) ry[i] = __ldg(Ay + k0 + 32 * i + lane);
    };
    fetch(0);
    for (int k0 = 0; k0 < terms; k0 += kAnchorStep) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            finite = finite && isfinite(rx[i]);
            if (32 * i + lane < kAnchorStep + 8) sx[32 * i + lane] = rx[i];
        }
#pragma unroll
        for (int i = 0; i < NY; ++i) {
            finite = finite && isfinite(ry[i]);
            sy[32 * i + lane + 4 * (4 * i + (lane >> 3))] = ry[i];
        }
        if (!__all_sync(kFullMask, finite)) break;
        if (k0 + kAnchorStep < terms) fetch(k0 + kAnchorStep);
        const double* x = sx + 8 + lc - lr;
        const double* y = sy + 12 * lr + lc;
        const int kn = min(kAnchorStep, (terms - k0 + 3) & ~3);
#pragma unroll 4
        for (int k = 0; k < kn; k += 4) {
            const double a = x[k];
            const int e = 12 * (k >> 3) + (k & 7);
#pragma unroll
            for (int p = 0; p < 4; ++p) mma_f64(c[p], a, y[96 * p + e]);
        }
    }
    if (__all_sync(kFullMask, finite)) {
        // c[p][h] is diagonal 8 (8p + 2 lc + h) + lr of the band
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            sq[8 * (8 * p + 2 * lc) + lr] = c[p][0];
            sq[8 * (8 * p + 2 * lc + 1) + lr] = c[p][1];
        }
    } else {
        tile_anchor_scalar<kAnchorChunk>(P.A, P.m, j0, gb, lane, area, sq + 8 * lane);
    }
    __syncwarp();
    double q[kTileR];
#pragma unroll
    for (int a = 0; a < kTileR; ++a) q[a] = sq[8 * lane + a];
    __syncwarp();
    const double mu0 = (double)P.m * __ldg(P.mean + j0);
#pragma unroll
    for (int a = 0; a < kTileR; ++a) nc[a] = __fma_rn(mu0, __ldg(P.mean + j0 + g0 + a), -q[a]);
}

// Persistent warps: each takes the next tile number from one global counter until
// the tile space is exhausted (no waiting on anything).
template <class F>
__device__ __forceinline__ void for_each_tile(const Fp32TileParams* series, int nseries, int64_t total,
                                              unsigned long long* counter, int lane, F tile) {
    for (;;) {
        unsigned long long t0 = 0;
        if (lane == 0) t0 = atomicAdd(counter, 1ull);
        const int64_t tt = (int64_t)__shfl_sync(kFullMask, t0, 0);
        if (tt >= total) break;
        // the series owning tile tt: last descriptor with tile_begin <= tt
        int lo = 0, hi = nseries - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (series[mid].tile_begin <= tt) lo = mid;
            else hi = mid - 1;
        }
        const Fp32TileParams P = series[lo];
        // local tile -> band and column segment (band pairs of nearly equal
        // tile counts); consecutive tiles are consecutive column segments of
        // one band, so tiles running together touch disjoint columns and rows
        int64_t band, seg;
        if (fp32_tile_of(P, tt - P.tile_begin + P.tile_skip, 32 * 8, band, seg))
            tile(P, band, seg);
    }
}

}  // namespace mpgpu
