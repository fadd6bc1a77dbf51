// Shared by the kernels that walk the FP32 form's tiles (32 * kTileR adjacent
// diagonals by K columns, one warp each): the FP32 join and the guarded form's
// FP64 pass.
#pragma once

#include "mp_common.cuh"
#include "mp_kernels.h"

namespace mpgpu {

constexpr int kTileR = 8;  // diagonals per lane

// FP64 re-anchor of a tile: minus the covariance at its first column j0 of the
// lane's diagonals g0 + a.  The series terms are staged in the warp's (not yet
// used) shared memory with coalesced loads, CHUNK terms at a time (anchor_bytes):
// the column's A[j0 + k] and the warp's rows A[j0 + gb + i], i < 32R + chunk, skewed
// by one double per 8 so that lanes reading rows 8 apart hit distinct banks.  Each
// lane then sums its R products in k order from shared memory.
template <int CHUNK>
__device__ __forceinline__ void tile_anchor(const Fp32TileParams& P, int64_t j0, int64_t gb, int64_t g0,
                                            int lane, char* area, double (&nc)[kTileR]) {
    constexpr int R = kTileR;
    double mu0 = (double)P.m * __ldg(P.mean + j0);
    double mr[R];
#pragma unroll
    for (int a = 0; a < R; ++a) mr[a] = __ldg(P.mean + j0 + g0 + a);
    double q[R];
#pragma unroll
    for (int a = 0; a < R; ++a) q[a] = 0.0;
    {
        static_assert(R % 8 == 0, "anchor row skew assumes lanes start on multiples of 8 rows");
        double* scol = reinterpret_cast<double*>(area);
        double* srow = scol + CHUNK;
        const double* Ac = P.A + j0;
        const double* Ar = P.A + j0 + gb;
        // lane's rows i = lane*R + t sit at srow[lane*(R + R/8) + t + t/8]
        const double* wl = srow + lane * (R + R / 8);
        for (int64_t kb0 = 0; kb0 < P.m; kb0 += CHUNK) {
            const int kc = (int)min((int64_t)CHUNK, P.m - kb0);
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
    for (int a = 0; a < R; ++a) nc[a] = __fma_rn(mu0, mr[a], -q[a]);
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
