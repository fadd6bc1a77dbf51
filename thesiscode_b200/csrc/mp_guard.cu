// Guarded FP32 form: FP64 tiles where the data is ill-conditioned for an FP32
// running sum.
//
// The FP32 recurrence's rounding error is relative to the covariance it
// carries, so a diagonal that passes, within one re-anchor interval, from
// windows of large norm (a level step on a walk, values straddling a constant
// stretch) to windows of far smaller norm carries a large absolute error into
// the small cells.  A window is a hazard when its norm is more than
// kGuardRatio times smaller than the largest norm among the K + 32R windows
// before it (that span covers every cell a tile can carry into it), or when it
// is flat.  Tiles whose column or row windows include a hazard are left out of
// the FP32 kernel and evaluated here with the same centred recurrence in FP64;
// both kernels min-merge into the same (ordered u, neighbour) keys.  On a
// plain random walk no window is a hazard.
#include <algorithm>
#include <atomic>

#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_tile.cuh"

namespace mpgpu {

namespace {

constexpr unsigned long long kNoKey = ~0ull;

__device__ __forceinline__ unsigned long long guard_key(float u, int64_t nb) {
    return ((unsigned long long)ord_f32(u) << 32) | (unsigned long long)nb;
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(kFullMask, v, o);
        v = w < v ? w : v;
    }
    return v;
}

// ---- FP64 tiles ---------------------------------------------------------------
// A warp walks the tile's columns with 8 diagonals per lane, as the FP32 join does
// (mp_join_fp32.cu): row terms in a shared-memory ring, groups of 8 rows, whose best
// keys sit beside them until the warp's lowest lane has met the row; a pass of 16
// columns first runs the recurrence with one more fused operation per cell, whose
// sign says whether the distance may be at or below the loosest bound among the
// rows' best keys and the columns' keys that the lane meets in the pass, and is
// evaluated again with the selection only when some lane has such a cell.  Every
// merge is a minimum of 64-bit keys, so the result does not depend on which cells
// the gate lets through beyond those that can lower a key.
//
// What bounds it: the FP64 pipe, 3 operations per cell and m per diagonal and tile
// for the anchor.  262,144 samples with 16 constant stretches, m = 1024, K = 512: 8
// ms (65.8 ms with every term and key read from global memory per cell).
constexpr int kCols = 16;    // columns per pass
constexpr int kGroups = 40;  // ring: groups of 8 rows; a pass reads 34, 2 more arrive
constexpr int kPad = 9;      // elements between groups: lanes 8 rows apart hit distinct banks
// The gate works in FP64: its margin covers the rounding of u to float.
constexpr double kSlack = 1e-6;
constexpr int kGuardSmem = 2 * kCols * 32 + kGroups * kPad * (16 + 8 + 8 + 8) + 2 * kCols * 4 + kGroups * 4;
static_assert(kGuardSmem % 16 == 0, "warps' areas stay 16-byte aligned");
static_assert(kAnchorBytes <= kGuardSmem, "anchor staging fits");
constexpr int kGuardWarps = 4;
constexpr int kGuardBlocksPerSm = 3;  // 8.2 ms against 8.8 at 2 (no spill) on the series above
__device__ __forceinline__ int wrap_group(int s) { return s < kGroups ? s : s - kGroups; }

// A key as it stands (merged meanwhile by other warps).
__device__ __forceinline__ unsigned long long ld_key(const unsigned long long* key) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(key));
    return v;
}
__device__ __forceinline__ unsigned key_bound(unsigned long long key) {
    return fp32_key_bound((unsigned)(key >> 32), false);
}

struct GuardSmem {
    double4* col;               // column terms df, dg, nn, 1 / nn, two buffers of kCols
    double2* dd;                // row terms df, dg, kPad per group
    double* nn;                 // ... and nn
    unsigned long long* best;   // best key per row
    unsigned long long* start;  // what it started from
    unsigned* cthr;             // column bounds (bit patterns), two buffers of kCols
    unsigned* gate;             // per group: the loosest of its rows' bounds
    __device__ __forceinline__ explicit GuardSmem(char* p) {
        col = reinterpret_cast<double4*>(p);
        dd = reinterpret_cast<double2*>(col + 2 * kCols);
        nn = reinterpret_cast<double*>(dd + kGroups * kPad);
        best = reinterpret_cast<unsigned long long*>(nn + kGroups * kPad);
        start = best + kGroups * kPad;
        cthr = reinterpret_cast<unsigned*>(start + kGroups * kPad);
        gate = cthr + 2 * kCols;
    }
    // Copies the terms of rows r .. r + 15 (two groups from slot s); zero past PL.
    __device__ __forceinline__ void stage_rows(const Fp32TileParams& P, int s, int64_t r, int lane) const {
        const int i = lane & 15, e = (s + (i >> 3)) * kPad + (i & 7);
        r += i;
        const bool in = r < P.PL;
        r = in ? r : 0;
        if (lane < 16) {
            cp_async8_or_zero(&dd[e].x, P.df + r, in);
            cp_async8_or_zero(nn + e, P.norm + r, in);
        } else {
            cp_async8_or_zero(&dd[e].y, P.dg + r, in);
        }
    }
    __device__ __forceinline__ unsigned group_gate(int s) const {
        unsigned g = 0;
#pragma unroll
        for (int k = 0; k < kTileR; ++k) g = max(g, key_bound(best[s * kPad + k]));
        return g;
    }
};

// A lane's window of 8 rows.
struct GuardWin {
    double df[8], dg[8], nn[8];
    __device__ __forceinline__ void load(const GuardSmem& sm, int s) {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const double2 x = sm.dd[s * kPad + a];
            df[a] = x.x;
            dg[a] = x.y;
            nn[a] = sm.nn[s * kPad + a];
        }
    }
};

// One pass without the selection: the result's sign bit is set when some cell of
// the lane may be at or below the bound, sn = 1 - bound less the slack (> 0).  On
// entry win holds the rows of the lane's first group, on return those of its third.
__device__ __forceinline__ int gate_pass(const GuardSmem& sm, int s1, int s2, const double4* col, double sn,
                                         GuardWin& win, double (&nc)[8]) {
    const double2 *d1 = sm.dd + s1 * kPad, *d2 = sm.dd + s2 * kPad;
    const double *n1 = sm.nn + s1 * kPad, *n2 = sm.nn + s2 * kPad;
    int t = 0;
#pragma unroll
    for (int b = 0; b < kCols; ++b) {
        const double4 cv = col[b];
        // nc * nn_r * nn_j < -sn  <=>  nc * nn_r + sn / nn_j < 0
        const double c = sn * cv.w;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int w = (b + a) % 8;
            t |= __double2hiint(__fma_rn(nc[a], win.nn[w], c));
            nc[a] = __fma_rn(-cv.x, win.dg[w], nc[a]);
            nc[a] = __fma_rn(win.df[w], -cv.y, nc[a]);
        }
        // row b gives way to row b + 8
        const double2 x = b < 8 ? d1[b] : d2[b - 8];
        win.df[b % 8] = x.x;
        win.dg[b % 8] = x.y;
        win.nn[b % 8] = b < 8 ? n1[b] : n2[b - 8];
    }
    return t;
}

// One pass with the selection, a loop over its columns.  EDGE: cell (column jr + b,
// diagonal g0 + d) exists iff d < ghi_rel and jr + b < min(lim0 - d, ncols), and
// every column selects; otherwise a column selects when some cell's distance is at
// or below `bound`.  Returns whether one did.
template <bool EDGE>
__device__ __forceinline__ bool select_pass(const Fp32TileParams& P, const GuardSmem& sm, int s0,
                                            const double4* col, const unsigned* cthr, double (&nc)[8],
                                            float bound, int lim0, int ncols, int ghi_rel, int jr, int64_t j0,
                                            int64_t g0, float ulim, int lane) {
    bool sel = false;
#pragma unroll 1
    for (int b = 0; b < kCols; ++b) {
        const int k = b % 8;  // cell d lies in element k + d of the groups sa, sb
        const int sa = wrap_group(s0 + b / 8), sb = wrap_group(sa + 1);
        const int e0 = sa * kPad + k, e1 = sb * kPad + k - 8;
        const double4 cv = col[b];
        float u[8], um = __builtin_huge_valf();
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            const int e = (k + d < 8 ? e0 : e1) + d;
            const double2 x = sm.dd[e];
            u[d] = (float)__fma_rn(nc[d], cv.z * sm.nn[e], 1.0);
            nc[d] = __fma_rn(-cv.x, x.y, nc[d]);
            nc[d] = __fma_rn(x.x, -cv.y, nc[d]);
            if (EDGE) {
                const int l = d < ghi_rel ? min(lim0 - d, ncols) : 0;
                if (jr + b >= l) u[d] = __builtin_huge_valf();
            }
            um = fminf(um, u[d]);
        }
        if (!EDGE && !__any_sync(kFullMask, um <= bound)) continue;
        sel = true;
        __syncwarp();  // rows move from lane to lane between columns
        const int64_t j = j0 + jr + b;
        unsigned long long ck = kNoKey;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (u[d] < ulim) {  // NaN (a flat window) never passes
                const int e = (k + d < 8 ? e0 : e1) + d;
                const unsigned long long kr = guard_key(u[d], j), kc = guard_key(u[d], j + g0 + d);
                if (kr < sm.best[e]) sm.best[e] = kr;
                ck = kc < ck ? kc : ck;
            }
        }
        if (__any_sync(kFullMask, um <= __uint_as_float(cthr[b]))) {
            ck = warp_min_u64(ck);
            if (lane == 0 && ck != kNoKey) atomicMin(P.key + j, ck);
        }
    }
    return sel;
}

__device__ void tile_guard(const Fp32TileParams& P, int64_t band, int64_t seg, int lane, const GuardSmem& sm) {
    constexpr int R = kTileR;
    const int64_t gb = P.g_lo + band * (int64_t)(32 * R);
    const int64_t g0 = gb + (int64_t)lane * R;
    const int64_t jmax = P.PL - gb;
    const int64_t j0 = seg * P.K;
    const int64_t j1 = min(j0 + P.K, jmax);
    if (j0 >= j1 || !fp32_tile_hazardous(P, gb, j0, j1, 32 * R)) return;
    const float ulim = (float)(1.0 + 1.0 / (double)P.m);
    const int ncols = (int)(j1 - j0);
    const int lim0 = (int)min(P.PL - g0 - j0, (int64_t)ncols + R);
    const int ghi_rel = (int)max(min(P.g_hi - g0, (int64_t)R), (int64_t)0);
    const int minlim = __reduce_min_sync(kFullMask, ghi_rel < R ? 0 : min(lim0 - (R - 1), ncols));

    double nc[R];  // m mean_j mean_r - sum A[j+k] A[r+k]  (= -covariance)
    tile_anchor(P, j0, gb, g0, lane, reinterpret_cast<char*>(sm.col), nc);

    // groups 0 .. 33 and the first pass's columns; from here on lanes 0 - 15 look
    // after rows, lanes 16 - 31 after columns
    const int64_t rb = j0 + gb;  // row of element 0 of group 0
    for (int i = 0; i < 17; ++i) sm.stage_rows(P, 2 * i, rb + 16 * i, lane);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int i = lane; i < 34 * R; i += 32) {
        const unsigned long long v = rb + i < P.PL ? ld_key(P.key + rb + i) : 0ull;
        sm.best[(i / R) * kPad + i % R] = v;
        sm.start[(i / R) * kPad + i % R] = v;
    }
    // a column's terms and bound; past PL they read as 0 and the gate stays shut
    auto put_column = [&](int buf, int i, double df, double dg, double nn, unsigned t) {
        sm.col[buf * kCols + i] = make_double4(df, dg, nn, __drcp_rn(nn));
        sm.cthr[buf * kCols + i] = t;
    };
    unsigned cgate = 0;
    if (lane < kCols) {
        const int64_t j = j0 + lane;
        const bool in = j < P.PL;
        cgate = in ? key_bound(ld_key(P.key + j)) : 0u;
        put_column(0, lane, in ? P.df[j] : 0.0, in ? P.dg[j] : 0.0, in ? P.norm[j] : 0.0, cgate);
    }
    cgate = __reduce_max_sync(kFullMask, cgate);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    sm.gate[lane] = sm.group_gate(lane);
    if (lane < 2) sm.gate[32 + lane] = sm.group_gate(32 + lane);
    __syncwarp();
    GuardWin win;
    win.load(sm, lane);

    const int64_t inc0 = lane < 16 ? rb + 34 * R + lane : j0 + lane;  // - 16 + kCols
    int s0 = lane;  // slot of the lane's first group
    int sf = 0;     // slot of the first group that the pass finishes
    int cb = 0;
    bool sel = false;
    int jr = 0;
    for (; jr < ncols; jr += kCols) {
        // what the next pass appends: 16 rows, 16 columns and their keys
        const int slot = wrap_group(sf + 34);
        sm.stage_rows(P, slot, rb + 34 * R + jr, lane);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const int64_t inc = inc0 + jr;
        unsigned long long key = 0ull;
        double cdf = 0.0, cdg = 0.0, cnn = 0.0;
        if (inc < P.PL) {
            key = ld_key(P.key + inc);
            if (lane >= 16) {
                cdf = __ldg(P.df + inc);
                cdg = __ldg(P.dg + inc);
                cnn = __ldg(P.norm + inc);
            }
        }
        const int s1 = wrap_group(s0 + 1), s2 = wrap_group(s0 + 2);
        const float bound =
            __uint_as_float(max(max(sm.gate[s0], sm.gate[s1]), max(sm.gate[s2], cgate)));
        const double4* col = sm.col + cb * kCols;
        const unsigned* cthr = sm.cthr + cb * kCols;
        const bool inside = jr + kCols <= minlim;
        bool open = !inside || sel;  // a pass after one that selected goes straight on
        if (!open) {
            double q0[8];
#pragma unroll
            for (int a = 0; a < 8; ++a) q0[a] = nc[a];
            const double sn = 1.0 - (double)bound - kSlack;
            const int t = gate_pass(sm, s1, s2, col, sn, win, nc);
            open = __any_sync(kFullMask, t < 0 || sn <= 0.0);
            if (open) {
#pragma unroll
                for (int a = 0; a < 8; ++a) nc[a] = q0[a];
            }
        }
        sel = false;
        if (open) {
            sel = inside ? select_pass<false>(P, sm, s0, col, cthr, nc, bound, lim0, ncols, ghi_rel, jr, j0, g0,
                                              ulim, lane)
                         : select_pass<true>(P, sm, s0, col, cthr, nc, bound, lim0, ncols, ghi_rel, jr, j0, g0,
                                             ulim, lane);
            win.load(sm, s2);
        }
        __syncwarp();
        // the pass's first two groups have met every lane: merge the rows that fell
        const unsigned f = inc < P.PL ? key_bound(key) : 0u;
        if (lane < 16) {
            const int e = (sf + (lane >> 3)) * kPad + (lane & 7);
            const unsigned long long v = sm.best[e];
            if (v < sm.start[e]) atomicMin(P.key + (rb + jr + lane), v);
            const int en = (slot + (lane >> 3)) * kPad + (lane & 7);
            sm.best[en] = key;
            sm.start[en] = key;
        } else {
            put_column(cb ^ 1, lane - 16, cdf, cdg, cnn, f);
        }
        const unsigned ga = __reduce_max_sync(kFullMask, lane < 8 ? f : 0u);
        const unsigned gc = __reduce_max_sync(kFullMask, (lane & 24) == 8 ? f : 0u);
        cgate = __reduce_max_sync(kFullMask, lane >= 16 ? f : 0u);
        if (lane == 0) {
            sm.gate[slot] = ga;
            sm.gate[slot + 1] = gc;
        }
        s0 = s2;
        if (sel) sm.gate[s0] = sm.group_gate(s0);  // bests of the groups still alive fell
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        sf = wrap_group(sf + 2);
        cb ^= 1;
    }

    // drain: rows of the next 32 groups
    for (int i = lane; i < 32 * R; i += 32) {
        const int e = wrap_group(sf + i / R) * kPad + i % R;
        const unsigned long long v = sm.best[e];
        if (v < sm.start[e]) atomicMin(P.key + (rb + jr + i), v);
    }
    __syncwarp();
}

// Same tile space and order as fp32_join_kernel; only hazard tiles do work.
__global__ void __launch_bounds__(32 * kGuardWarps, kGuardBlocksPerSm)
    fp64_guard_kernel(const Fp32TileParams* __restrict__ series, int nseries, int64_t total,
                      unsigned long long* __restrict__ counter) {
    extern __shared__ __align__(128) char smem_guard[];
    const int lane = threadIdx.x & 31;
    const GuardSmem sm(smem_guard + (threadIdx.x >> 5) * kGuardSmem);
    for_each_tile(series, nseries, total, counter, lane,
                  [&](const Fp32TileParams& P, int64_t band, int64_t seg) {
                      if (P.hazard) tile_guard(P, band, seg, lane, sm);
                  });
}

}  // namespace

// Van Herk / Gil-Werman sliding minimum, part 1: prefix and suffix minima of
// the inverse norms within blocks of `blk` windows (NaN, a flat window, is
// ignored by fmin).
__global__ void hazard_block_minima_kernel(const double* __restrict__ nn, int64_t PL, int64_t blk,
                                           double* __restrict__ pre, double* __restrict__ suf) {
    hazard_block_minima(nn, PL, blk, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, pre, suf);
}

// Part 2: flag[w + 1] = 1 when window w is a hazard: flat, or its inverse norm
// exceeds kGuardRatio times the smallest inverse norm among windows
// [w - look, w] (look = blk - 1).  flag[0] = 0; an inclusive scan then turns
// flag into prefix counts.
__global__ void hazard_flags_kernel(const double* __restrict__ nn, const double* __restrict__ pre,
                                    const double* __restrict__ suf, int64_t PL, int64_t blk,
                                    int* __restrict__ flag) {
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w <= PL;
         w += (int64_t)gridDim.x * blockDim.x) {
        if (w == PL) {
            flag[0] = 0;
            continue;
        }
        flag[w + 1] = hazard_flag(nn, pre, suf, blk, w);
    }
}

// FP64 recurrence terms, the FP32 records' formulas without the rounding to
// float: df[i] = (A[i+m] - A[i]) / 2, dg[i] = (A[i+m] - mean[i+1]) + (A[i] - mean[i]).
__global__ void guard_terms_kernel(const double* __restrict__ A, int64_t m, int64_t PL,
                                   const double* __restrict__ mean, double* __restrict__ df,
                                   double* __restrict__ dg) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < PL;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (i + 1 < PL) {
            const double xin = A[i + m], xout = A[i];
            df[i] = (xin - xout) * 0.5;
            dg[i] = (xin - mean[i + 1]) + (xout - mean[i]);
        } else {
            df[i] = 0.0;
            dg[i] = 0.0;
        }
    }
}

// ---- near-duplicate pass ----------------------------------------------------
// Windows whose best FP32 u lies below the FP32 resolution floor (u formed by
// cancellation carries an absolute error of ~1e-7..1e-6) are collected, their
// keys reset, and every pair among them recomputed exactly: a near-duplicate's
// best partner has a tiny u too, so it is in the same set.

__global__ void neardup_collect_kernel(const unsigned long long* __restrict__ key, int64_t PL,
                                       float tau, unsigned long long init, int* __restrict__ list,
                                       int* __restrict__ count, int cap) {
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < PL;
         w += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long k = key[w];
        if (k >= init) continue;  // no neighbour
        if (unord_f32((unsigned)(k >> 32)) < tau) {
            const int i = atomicAdd(count, 1);
            if (i < cap) list[i] = (int)w;
        }
    }
}

__global__ void neardup_reset_kernel(const int* __restrict__ list, int count,
                                     unsigned long long* __restrict__ key, unsigned long long init) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        key[list[i]] = init;
}

// Tile (ti, tj) of the list x list pair square, 32 x 32 pairs, 2 x 2 per
// thread: centred FP64 dot products, u = 1 - dot * nn_w * nn_v, min-merged
// into the row window's key (the square holds both orders of every pair).
__global__ void __launch_bounds__(256) neardup_pairs_kernel(const NearDupParams P) {
    constexpr int TB = 32, KC = 32;
    __shared__ double sr[TB][KC + 1];
    __shared__ double sc[TB][KC + 1];
    __shared__ unsigned long long rmin[TB][16];
    const int64_t nt = (P.count + TB - 1) / TB;
    const int64_t ti = blockIdx.x / nt, tj = blockIdx.x % nt;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int64_t k0 = 0; k0 < P.m; k0 += KC) {
        __syncthreads();
        for (int e = threadIdx.x; e < TB * KC; e += blockDim.x) {
            const int q = e / KC, kk = e % KC;
            const int64_t k = k0 + kk;
            const int64_t ir = ti * TB + q, ic = tj * TB + q;
            double vr = 0.0, vc = 0.0;
            if (k < P.m && ir < P.count) {
                const int64_t w = P.list[ir];
                vr = P.A[w + k] - P.mean[w];
            }
            if (k < P.m && ic < P.count) {
                const int64_t v = P.list[ic];
                vc = P.A[v + k] - P.mean[v];
            }
            sr[q][kk] = vr;
            sc[q][kk] = vc;
        }
        __syncthreads();
        const int kn = (int)min((int64_t)KC, P.m - k0);
        for (int kk = 0; kk < kn; ++kk) {
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    acc[a][c] = __fma_rn(sr[ty * 2 + a][kk], sc[tx * 2 + c][kk], acc[a][c]);
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int64_t ir = ti * TB + ty * 2 + a;
        unsigned long long best = kNoKey;
        if (ir < P.count) {
            const int64_t w = P.list[ir];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int64_t ic = tj * TB + tx * 2 + c;
                if (ic >= P.count) continue;
                const int64_t v = P.list[ic];
                const int64_t g = w > v ? w - v : v - w;
                if (g < P.g_lo || g >= P.g_hi) continue;
                const double u = __fma_rn(-acc[a][c], P.norm[w] * P.norm[v], 1.0);
                const float fu = (float)u;
                if (fu < P.ulim) {
                    const unsigned long long kk = guard_key(fu, v);
                    best = kk < best ? kk : best;
                }
            }
        }
        rmin[ty * 2 + a][tx] = best;
    }
    __syncthreads();
    if (threadIdx.x < TB) {
        const int64_t ir = ti * TB + threadIdx.x;
        unsigned long long best = kNoKey;
        for (int x = 0; x < 16; ++x) best = rmin[threadIdx.x][x] < best ? rmin[threadIdx.x][x] : best;
        if (ir < P.count && best != kNoKey) atomicMin(P.key + P.list[ir], best);
    }
}

template <int R>
void launch_fp64_guard(const Fp32TileParams* series_dev, int nseries, int64_t total,
                       unsigned long long* counter, cudaStream_t s) {
    static_assert(R == kTileR, "the tile kernel is laid out for 8 diagonals per lane");
    // per-device attribute, idempotent: see launch_fp32_join
    static std::atomic<unsigned long long> configured{0};
    constexpr int smem = kGuardWarps * kGuardSmem;
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(fp64_guard_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        configured.fetch_or(bit, std::memory_order_release);
    }
    const int64_t want = (total + kGuardWarps - 1) / kGuardWarps;
    const int64_t blocks = std::min<int64_t>(want, (int64_t)sm_count() * kGuardBlocksPerSm);
    if (blocks > 0)
        fp64_guard_kernel<<<(unsigned)blocks, 32 * kGuardWarps, smem, s>>>(series_dev, nseries, total, counter);
}

template void launch_fp64_guard<8>(const Fp32TileParams*, int, int64_t, unsigned long long*,
                                   cudaStream_t);

}  // namespace mpgpu
