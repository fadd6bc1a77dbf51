// FP64 diagonal-band join: the reference's SCRIMP recurrence evaluated with
// the reference's own per-cell arithmetic, one warp per band of 32*R
// adjacent diagonals.
//
// Reference: eval_diag_block_triangle, AVX2 branch
// (scrimppp/src/kernels.cpp:170-307), driven over blocks of blocklen
// diagonals by ScrimpVertBlocked (scrimppp/src/ScrimpVertBlocked.cpp:139-168).
// Per cell (column j, diagonal g, row r = j + g):
//   4-wide part : score = fma(QT, s_r*s_j, -(mu_j*mu_r))
//                 QT    = fma(-A[r], A[j], fma(A[r+m], A[j+m], QT))
//   remainder   : score = QT*(s_r*s_j) - mu_r*mu_j, QT = (QT + A[r+m]*A[j+m]) - A[r]*A[j]
// (every product and sum separately rounded).  A cell is in the remainder
// iff its offset in the reference block, delta, is >= 4*floor(cnt/4) with
// cnt = min(blocklen, T - j); for a diagonal that is only its last
// 3 - delta%4 cells (or all of it when delta >= blocklen & ~3).
//
// Work layout (B200): lane l of a warp owns diagonals g0 + a, a < R,
// g0 = band start + l*R; all lanes walk the same column j.  Per step a lane
// evaluates R cells; no two of a step's 32*R cells share a row.  The best cell
// of every row alive in the band sits in the warp's shared memory until the
// warp's lowest lane has met the row; a column is complete in one step.
// Finished rows and columns go to global memory as 64-bit max reductions into
// one of several key shards.  One resident wave of warps takes the bands
// from a list (fp64_band_of).
//
// Selection thresholds: every merge also raises a per-entry threshold to a
// value just below the merged score (fp64_threshold_below: the margin is wider
// than the index key's resolution).  A row's best cell starts at its row's
// threshold with no source.  A cell that exceeds neither its row's best nor its
// column's threshold can raise neither key of its row or column (its score is
// below a score already merged there, by more than the index key resolves), so
// the result is the same as selecting every cell.  Thresholds are read as they
// stand (a stale one is only a lower bound), so the arithmetic and the keys --
// and therefore the output -- do not depend on timing.
//
// Bands of one wave run side by side, and a row's first candidates come from
// the band whose diagonals reach it first.  If the wave holds the longest bands
// only, every row past its last band is new to all of them: the band next to
// those rows selects in nearly every step, the ones behind catch up with it, and
// soon the whole wave selects (n = 1,048,576: 16% of the steps had a cell above
// its row's best).  So the first wave takes every spread-th band of the whole
// list; the bands between them then meet rows whose bests are nearly final.
//
// Passes inside the 4-wide part test in integers, once per kU * R columns: a lane
// takes the maximum of its scores' high words and compares it with the smallest
// high word among the best scores of the rows and the thresholds of the columns
// that it meets in the pass (fp64_gate; high words order like non-negative
// doubles, and a negative bound opens the gate).  When some lane of the warp
// passes, the pass is evaluated again with the selection.  That takes R/2 integer
// maxima per column in place of 2R FP64 compares and two votes, and no branch
// between the columns.
//
// What bounds it: the FP64 pipe takes a warp's instruction every 2.2 cycles, 5
// per cell (40 of a step's 62 instructions at R = 8); other instructions cost it
// about 0.7 cycles each.  n = 1,048,576, m = 256: 262 ms, from 441 ms with the
// selection tested per step in FP64 and the bands in order of length (spread
// alone: 269 ms, with the gate per step).  3 CTAs of 4 warps per SM at 168
// registers spill and run at 273 ms.
#include <float.h>
#include <limits.h>

#include <algorithm>
#include <atomic>

#include "mp_common.cuh"
#include "mp_kernels.h"

namespace mpgpu {

namespace {

// A 32-byte record of the warp's shared-memory ring (16-byte aligned halves).
__device__ __forceinline__ double4 ring_rec(const char* p) {
    const double2 a = *reinterpret_cast<const double2*>(p);
    const double2 b = *reinterpret_cast<const double2*>(p + 16);
    return make_double4(a.x, a.y, b.x, b.y);
}

// Asynchronous 16-byte copy global -> shared through L2 only (both addresses
// 16-byte aligned).
__device__ __forceinline__ void cp_async16(char* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
// A threshold as it stands (other warps raise it with atomics meanwhile; any
// value it has held is a valid lower bound).
__device__ __forceinline__ double ld_thr(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void flush_fp64(const Fp64BandParams& P, int shard, int64_t slot,
                                           double score, int64_t neighbour) {
    unsigned long long* ke = P.kexact + (int64_t)shard * P.key_stride + slot;
    unsigned long long* ki = P.kidx + (int64_t)shard * P.key_stride + slot;
    atomicMax(ke, ord_f64(score));
    atomicMax(ki, idx_key_f64(score, P.m, (unsigned long long)neighbour, P.idx_bits, P.key_vlo));
    // thresholds only ever hold non-negative values above their -DBL_MAX
    // start, where the signed 64-bit pattern orders like the double
    const double t = fp64_threshold_below(score, P.m, P.thr_eps, P.thr_tiny);
    if (t >= 0.0) atomicMax(reinterpret_cast<long long*>(P.thr + slot), __double_as_longlong(t));
}

// A bound's high word for the integer gate: scores at or above a non-negative
// bound have a high word at or above its high word (as signed integers); a
// negative bound lets every cell through.
__device__ __forceinline__ int fp64_gate(double bound) {
    const int h = __double2hiint(bound);
    return h < 0 ? INT_MIN : h;
}

// One warp's shared memory.  Rows of the band go in groups of R (row t of the
// tile, counted from its first column's row on the band's first diagonal, is
// element t % R of group t / R); kGroups slots of R rows form a ring, in which
// chunk c reads groups c .. c + 32; a pass of kU chunks copies in the next kU
// groups meanwhile.  Every
// array is padded by one element per group, so that lanes reading the same
// element of consecutive groups hit distinct banks (a multiple of 8 groups, so
// that a wrap keeps that for the 16-byte halves of the records).
constexpr int kGroups = 40;
constexpr int kU = 2;  // chunks per pass
static_assert(kGroups % kU == 0 && kGroups >= 32 + 2 * kU, "a pass's incoming groups fit the ring");
__device__ __forceinline__ int wrap_group(int s) { return s < kGroups ? s : s - kGroups; }
template <int R>
struct BandSmem {
    static constexpr int kRecStride = 32 * R + 16;  // bytes of a group's records
    static constexpr int kUsed = kGroups * kRecStride + 2 * 32 * R * kU +
                                 kGroups * (R + 1) * (int)(sizeof(double) + sizeof(int)) +
                                 2 * R * kU * (int)sizeof(double) + kGroups * (int)sizeof(int);
    static constexpr int kBytes = (kUsed + 15) / 16 * 16;  // warps' areas stay aligned
    char* rec;     // row records
    char* col;     // column records, two buffers of kU * R
    double* best;  // best score of each row (its threshold while src < 0)
    double* cthr;  // column thresholds, two buffers of kU * R
    int* src;      // its column, -1: none yet
    int* gate;     // per group: smallest gate among the rows' best scores
    __device__ __forceinline__ BandSmem(char* p) {
        rec = p;
        p += kGroups * kRecStride;
        col = p;
        p += 2 * 32 * R * kU;
        best = reinterpret_cast<double*>(p);
        p += kGroups * (R + 1) * sizeof(double);
        cthr = reinterpret_cast<double*>(p);
        p += 2 * R * kU * sizeof(double);
        src = reinterpret_cast<int*>(p);
        p += kGroups * (R + 1) * sizeof(int);
        gate = reinterpret_cast<int*>(p);
    }
    // smallest gate among the R rows of the group in slot s
    __device__ __forceinline__ int group_gate(int s) const {
        int g = INT_MAX;
#pragma unroll
        for (int k = 0; k < R; ++k) g = min(g, fp64_gate(best[s * (R + 1) + k]));
        return g;
    }
};

// The column's best cell over the warp, from two REDUX instructions (high, then
// low word of the ordered score; ties go to the smallest diagonal); the winning
// lane merges it.
template <int R>
__device__ __forceinline__ void select_column(const Fp64BandParams& P, int shard, unsigned j,
                                              const double (&sc)[R], int64_t g0, int lane) {
    // lane's best cell of the column: pairwise tree, left wins ties.  A NaN
    // cell (a constant window) never selects under the reference's '>'; as
    // -DBL_MAX it also cannot hide the cell it is paired with in the tree.
    double cb[R];
    int ca[R];
#pragma unroll
    for (int a = 0; a < R; ++a) {
        cb[a] = sc[a] == sc[a] ? sc[a] : -DBL_MAX;
        ca[a] = a;
    }
#pragma unroll
    for (int w = 1; w < R; w *= 2)
#pragma unroll
        for (int a = 0; a + w < R; a += 2 * w)
            if (cb[a + w] > cb[a]) {
                cb[a] = cb[a + w];
                ca[a] = ca[a + w];
            }
    const double cbest = cb[0];
    const unsigned long long key = (cbest > P.floor) ? ord_f64(cbest) : 0ull;
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(kFullMask, hi);
    const unsigned mlo = __reduce_max_sync(kFullMask, hi == mhi ? lo : 0u);
    const bool top = (hi == mhi) && (lo == mlo) && (mhi != 0u);
    const unsigned tops = __ballot_sync(kFullMask, top);
    if (top && (tops & ((1u << lane) - 1u)) == 0u)
        flush_fp64(P, shard, j + P.col_key_off, cbest, j + g0 + ca[0] + P.row_nb_off);
}

// Selection of one column step: every cell above its row's best replaces it
// (strict '>', the reference's rule; a step's cells lie in distinct rows), and
// a column with a cell above its threshold tc is reduced over the warp.  Cell a
// of column b is element b + a of the lane's two groups, in slots s0 and s1.
template <int R>
__device__ __forceinline__ void select_step(const Fp64BandParams& P, int shard, int b, unsigned j,
                                            const double (&sc)[R], const BandSmem<R>& sm, int s0,
                                            int s1, double tc, int64_t gb, int lane) {
    __syncwarp();  // rows move from lane to lane between steps
    bool col = false;
#pragma unroll
    for (int a = 0; a < R; ++a) {
        const int e = b + a < R ? s0 * (R + 1) + b + a : s1 * (R + 1) + b + a - R;
        if (sc[a] > sm.best[e]) {
            sm.best[e] = sc[a];
            sm.src[e] = (int)j;
        }
        col |= sc[a] > tc;
    }
    if (__any_sync(kFullMask, col)) select_column<R>(P, shard, j, sc, gb + lane * R, lane);
}

// One chunk = R consecutive columns, in one of three ways:
//   kGate    only cells of the reference's 4-wide (fused) part, no selection:
//            returns the largest high word of the lane's scores
//   kSelect  the same cells again with the selection, for a chunk whose gate
//            opened: per step behind the gate
//   kEdge    any cells, each with its own geometry; every step selects
// On entry rwin holds the records of the lane's first group, on return those of
// its second.
// (sel: set when a step selected).
enum ChunkWay { kGate, kSelect, kEdge };
template <int R, ChunkWay WAY>
__device__ __forceinline__ int chunk_fp64(const Fp64BandParams& P, int shard, unsigned jc,
                                          const BandSmem<R>& sm, int s0, int s1,
                                          const char* col, const double* cthr,
                                          double4 (&rwin)[R], double (&qt)[R], int gate,
                                          unsigned geo, int64_t gb, int lane, bool& sel) {
    const int len0 = (int)(P.Tbase - gb) - lane * R;  // columns of the lane's first diagonal
    int top = INT_MIN;
    const char* rec1 = sm.rec + s1 * BandSmem<R>::kRecStride;
    double4 cv = ring_rec(col);
#pragma unroll
    for (int b = 0; b < R; ++b) {
        const unsigned j = jc + b;
        double4 cn = cv;
        if (b + 1 < R) cn = ring_rec(col + 32 * (b + 1));
        double sc[R];
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const double4 rv = rwin[(b + a) % R];
            // the window moves on: element b + R replaces element b
            if (a == 0) rwin[b] = ring_rec(rec1 + 32 * b);
            double score = -DBL_MAX;
            const unsigned code = (geo >> (4 * a)) & 15u;
            if (WAY != kEdge || (code != 15u && (int64_t)j < len0 - a)) {
                const double ss = __dmul_rn(rv.z, cv.z);
                if (WAY != kEdge || (code != 7u && (int64_t)j <= len0 - a - 4 + (int)code)) {
                    // 4-wide part of the reference kernel (kernels.cpp:206-225)
                    const double mm = __dmul_rn(cv.w, rv.w);
                    score = __fma_rn(qt[a], ss, -mm);
                    qt[a] = __fma_rn(-rv.x, cv.x, __fma_rn(rv.y, cv.y, qt[a]));
                } else {
                    // scalar remainder (kernels.cpp:282-289), no fusion
                    score = __dsub_rn(__dmul_rn(qt[a], ss), __dmul_rn(rv.w, cv.w));
                    qt[a] = __dsub_rn(__dadd_rn(qt[a], __dmul_rn(rv.y, cv.y)),
                                      __dmul_rn(rv.x, cv.x));
                }
            }
            sc[a] = score;
        }
        cv = cn;
        if (WAY != kEdge) {
            if (WAY == kSelect) top = INT_MIN;
            if (R == 1) top = max(top, __double2hiint(sc[0]));
#pragma unroll
            for (int a = 0; a + 1 < R; a += 2)
                top = __vimax3_s32(top, __double2hiint(sc[a]), __double2hiint(sc[a + 1]));
        }
        if (WAY == kEdge || (WAY == kSelect && __any_sync(kFullMask, top >= gate))) {
            select_step<R>(P, shard, b, j, sc, sm, s0, s1, cthr[b], gb, lane);
            sel = true;
        }
    }
    return top;
}

template <int R>
__device__ __forceinline__ void band_fp64(const Fp64BandParams& P, int64_t band, int lane,
                                          int shard, const BandSmem<R>& sm) {
    constexpr int RS = BandSmem<R>::kRecStride;
    const int64_t gb = P.g_lo + band * (int64_t)(32 * R);
    const int64_t g0 = gb + (int64_t)lane * R;
    const int jmax = (int)(P.Tbase - gb);  // length of the band's longest diagonal
    if (jmax <= 0) return;

    // Diagonal g has len = Tbase - g columns; with delta its offset in its block,
    // its last column of the reference's 4-wide part is len - 4 + delta % 4, or
    // none when delta >= B & ~3.  geo holds delta % 4 (or 7) of the lane's
    // diagonals, 15 for one past g_hi, as nibbles: only the chunks near a
    // diagonal's end read them.  A diagonal past g_hi carries -inf, which stays
    // below every bound, so it does not cost the band its branch-free chunks.
    double qt[R];
    unsigned geo = 0;
    int minpsw = INT_MAX;
#pragma unroll
    for (int a = 0; a < R; ++a) {
        const int64_t g = g0 + a;
        unsigned code = 15;
        qt[a] = -__longlong_as_double(0x7ff0000000000000ll);
        if (g < P.g_hi) {
            const int64_t delta = (g - P.blk_origin) % P.B;
            qt[a] = P.qt0[g - P.g_lo];
            code = delta < (P.B & ~3ll) ? (unsigned)(delta & 3) : 7u;
            minpsw = min(minpsw, code == 7u ? -1 : (int)(P.Tbase - g) - 4 + (int)code);
        }
        geo |= code << (4 * a);
    }
    minpsw = __reduce_min_sync(kFullMask, minpsw);

    // Groups 0 .. 32 + kU - 1 and the first pass's columns.  In a pass of kU
    // chunks, lanes 0 - 15 bring in the next rows' thresholds, lanes 16 - 31 the
    // next columns': part = lane % 16.
    const int part = lane & 15;
    const bool isrow = lane < 16;
    const uint4* rsrc = reinterpret_cast<const uint4*>(P.rowrec + gb);
    const uint4* crec = reinterpret_cast<const uint4*>(P.colrec);
    const double* tsrc = P.thr + gb + P.row_key_off;  // threshold of row t
    const double* csrc = P.thr + P.col_key_off;       // threshold of column j
    for (int i = lane; i < (32 + kU) * 2 * R; i += 32)
        *reinterpret_cast<uint4*>(sm.rec + (i / (2 * R)) * RS + 16 * (i % (2 * R))) =
            __ldg(rsrc + i);
    for (int i = lane; i < (32 + kU) * R; i += 32) {
        sm.best[(i / R) * (R + 1) + i % R] = ld_thr(tsrc + i);
        sm.src[(i / R) * (R + 1) + i % R] = -1;
    }
    if (lane < 2 * R * kU) *reinterpret_cast<uint4*>(sm.col + 16 * lane) = __ldg(crec + lane);
    int cgate = INT_MAX;
    if (lane < R * kU) {
        const double t = ld_thr(csrc + lane);
        sm.cthr[lane] = t;
        cgate = fp64_gate(t);
    }
    cgate = __reduce_min_sync(kFullMask, cgate);
    __syncwarp();
    sm.gate[lane] = sm.group_gate(lane);
    if (lane < kU) sm.gate[32 + lane] = sm.group_gate(32 + lane);
    __syncwarp();
    // register window of row records: slot (k mod R) holds element k of the
    // lane's first group
    double4 rwin[R];
#pragma unroll
    for (int k = 0; k < R; ++k) rwin[k] = ring_rec(sm.rec + lane * RS + 32 * k);

    // what the lane copies in next: records of groups c + 32 + kU .. and of the
    // next pass's columns, and their thresholds
    const uint4* nrow = rsrc + (32 + kU) * 2 * R + lane;
    const uint4* ncol = crec + kU * 2 * R + lane;
    const double* nthr = isrow ? tsrc + (32 + kU) * R + part : csrc + kU * R + part;
    int s0 = lane;  // slot of the lane's first group
    int sf = 0;     // slot of group c, the first that the pass finishes
    int cbuf = 0;
    bool sel = false;
    for (unsigned jc = 0; jc < (unsigned)jmax; jc += kU * R) {
        const int sn = wrap_group(sf + 32 + kU);  // slots of the incoming groups (kU divides kGroups)
        double t = 0.0;
        if (lane < 2 * R * kU) {
            cp_async16(sm.rec + (sn + lane / (2 * R)) * RS + 16 * (lane % (2 * R)), nrow);
            cp_async16(sm.col + (cbuf ^ 1) * (32 * R * kU) + 16 * lane, ncol);
        }
        if (part < R * kU) t = ld_thr(nthr);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        nrow += kU * 2 * R;
        ncol += kU * 2 * R;
        nthr += kU * R;
        int gate = cgate;
#pragma unroll
        for (int u = 0; u <= kU; ++u) gate = min(gate, sm.gate[wrap_group(s0 + u)]);
        const char* col = sm.col + cbuf * (32 * R * kU);
        const double* cthr = sm.cthr + cbuf * (R * kU);
        if ((int64_t)jc + (kU * R - 1) <= minpsw) {
            bool open = sel;  // a pass after one that selected goes straight to selecting
            if (!open) {
                double q0[R];
#pragma unroll
                for (int a = 0; a < R; ++a) q0[a] = qt[a];
                int top = INT_MIN;
#pragma unroll 1
                for (int u = 0; u < kU; ++u)
                    top = max(top, chunk_fp64<R, kGate>(P, shard, jc + u * R, sm, wrap_group(s0 + u), wrap_group(s0 + u + 1),
                                                        col + u * 32 * R, cthr + u * R, rwin, qt, gate, geo, gb, lane, open));
                open = __any_sync(kFullMask, top >= gate);
                if (open) {
#pragma unroll
                    for (int a = 0; a < R; ++a) {
                        qt[a] = q0[a];
                        rwin[a] = ring_rec(sm.rec + s0 * RS + 32 * a);
                    }
                }
            }
            sel = false;
            if (open) {
#pragma unroll 1
                for (int u = 0; u < kU; ++u)
                    chunk_fp64<R, kSelect>(P, shard, jc + u * R, sm, wrap_group(s0 + u), wrap_group(s0 + u + 1),
                                           col + u * 32 * R, cthr + u * R, rwin, qt, gate, geo, gb, lane, sel);
            }
        } else {
            sel = true;
#pragma unroll 1
            for (int u = 0; u < kU; ++u)
                chunk_fp64<R, kEdge>(P, shard, jc + u * R, sm, wrap_group(s0 + u), wrap_group(s0 + u + 1),
                                     col + u * 32 * R, cthr + u * R, rwin, qt, gate, geo, gb, lane, sel);
        }
        __syncwarp();
        // groups c .. c + kU - 1 have met every lane: merge their rows
        if (lane < R * kU) {
            const int e = (sf + lane / R) * (R + 1) + lane % R;
            const int j = sm.src[e];
            if (j >= 0) {
                const double s = sm.best[e];
                if (s > P.floor) flush_fp64(P, shard, jc + gb + lane + P.row_key_off, s, j + P.col_nb_off);
            }
        }
        // the incoming groups and columns begin at their thresholds
        if (part < R * kU) {
            if (isrow) {
                const int e = (sn + part / R) * (R + 1) + part % R;
                sm.best[e] = t;
                sm.src[e] = -1;
            } else {
                sm.cthr[(cbuf ^ 1) * (R * kU) + part] = t;
            }
        }
        const int x = part < R * kU ? fp64_gate(t) : INT_MAX;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int g = __reduce_min_sync(kFullMask, isrow && part / R == u ? x : INT_MAX);
            if (lane == 0) sm.gate[sn + u] = g;
        }
        cgate = __reduce_min_sync(kFullMask, isrow ? INT_MAX : x);
        s0 = wrap_group(s0 + kU);
        if (sel) sm.gate[s0] = sm.group_gate(s0);  // best scores of groups c + kU .. c + kU + 31 rose
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        sf = wrap_group(sf + kU);
        cbuf ^= 1;
    }

    // drain: rows of groups c .. c + 31 (the last chunk's second groups)
    const int64_t tend = ((int64_t)jmax + kU * R - 1) / (kU * R) * (kU * R);  // row t of group c
    for (int i = lane; i < 32 * R; i += 32) {
        const int s = wrap_group(sf + i / R);
        const int e = s * (R + 1) + i % R;
        const int j = sm.src[e];
        if (j >= 0) {
            const double v = sm.best[e];
            if (v > P.floor) flush_fp64(P, shard, tend + gb + i + P.row_key_off, v, j + P.col_nb_off);
        }
    }
    __syncwarp();

    if (P.qt_out) {
#pragma unroll
        for (int a = 0; a < R; ++a)
            if (g0 + a < P.g_hi) P.qt_out[g0 + a - P.g_lo] = qt[a];
    }
}

template <int R>
constexpr int fp64_smem_bytes() {
    return kFp64WarpsPerBlock * BandSmem<R>::kBytes;
}

template <int R>
__global__ void __launch_bounds__(32 * kFp64WarpsPerBlock, R == 8 ? 2 : 4)
    fp64_band_kernel(const Fp64BandParams P) {
    extern __shared__ __align__(128) char smem_fp64[];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const BandSmem<R> sm(smem_fp64 + w * BandSmem<R>::kBytes);
    // One resident wave of W warps takes the bands by rank (fp64_band_of): warp
    // w starts with rank w, later ranks come from one counter (no waiting on
    // anything).
    const int64_t wid = (int64_t)blockIdx.x * kFp64WarpsPerBlock + w;
    const int shard = (int)(wid % P.shards);
    for (int64_t rank = wid; rank < P.nbands;) {
        band_fp64<R>(P, fp64_band_of(rank, P.nbands, P.spread), lane, shard, sm);
        unsigned next = 0;
        if (lane == 0) next = atomicAdd(P.counter, 1u);
        rank = (int64_t)gridDim.x * kFp64WarpsPerBlock + __shfl_sync(kFullMask, next, 0);
    }
}

}  // namespace

template <int R>
void launch_fp64_band(const Fp64BandParams& Q, cudaStream_t s) {
    constexpr int smem = fp64_smem_bytes<R>();
    // per-device attribute and occupancy, idempotent: see launch_fp32_join
    static std::atomic<unsigned long long> configured{0};
    static std::atomic<int> resident[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(fp64_band_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fp64_band_kernel<R>,
                                                          32 * kFp64WarpsPerBlock, smem) != cudaSuccess ||
            per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        resident[dev & 63].store(per_sm, std::memory_order_relaxed);
        configured.fetch_or(bit, std::memory_order_release);
    }
    // one resident wave, fewer CTAs when there are fewer bands than warps
    const int64_t wave = (int64_t)sm_count() * resident[dev & 63].load(std::memory_order_relaxed);
    const int64_t want = (Q.nbands + kFp64WarpsPerBlock - 1) / kFp64WarpsPerBlock;
    const int64_t blocks = std::min<int64_t>(want, wave);
    if (blocks <= 0) return;
    Fp64BandParams P = Q;
    P.spread = (P.nbands + blocks * kFp64WarpsPerBlock - 1) / (blocks * kFp64WarpsPerBlock);
    cudaMemsetAsync(P.counter, 0, sizeof(unsigned), s);
    fp64_band_kernel<R><<<(unsigned)blocks, 32 * kFp64WarpsPerBlock, smem, s>>>(P);
}

template void launch_fp64_band<1>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<2>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<4>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<8>(const Fp64BandParams&, cudaStream_t);

}  // namespace mpgpu
