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
// Passes (16 columns) inside the 4-wide part only look for a cell that could select:
// a column's gate is the score in the form s' (q s - w W'), W' = w' / s', whose last
// product is taken once for the lane's R cells: 4 FP64 operations per cell in place of
// 5.  Its high word is compared with those of the column's threshold and of the
// smallest best score among the R rows (fp64_gate and the functions beside it: the
// bounds lie below by more than the two forms' rounding differs).  When some lane
// of the warp passes, the pass is evaluated again with the reference's arithmetic and
// the selection.  High words take R/2 integer maxima and two additions per column
// where doubles took 2R compares, and no branch between the columns.
//
// How often a gate opens depends on the data: noisy patterns, short windows and series of few
// levels have rows of unlike best scores side by side, and the smallest of R opens many
// passes in which no cell selects.  So whole bands (WHOLE) back off: after gates that opened
// in a row, and after a pass that selected, passes go straight to the reference's
// arithmetic, 4 columns at a time, each cell tested against its own row's best
// (test_chunk); only columns from such a cell on, to the end of 8, are evaluated with the
// selection.  300,000 samples: noisy sine, m = 64 61 -> 47 ms (46 with every step tested in
// FP64), half NaN 117 -> 44 (46), steps of 150 samples, m = 256 97 -> 77 (67); 280,000, m = 16,
// walk 81 -> 45 (43), sine 106 -> 44 (43).  Tiles, short and young, select more of what they
// test, and evaluate an open pass with the selection throughout (n = 65,536: 1.58 ms;
// as whole bands do 1.77).
//
// What bounds it: the FP64 pipe takes a warp's instruction every 2.2 cycles, 4
// per cell (33 of a step's 60 instructions at R = 8); other instructions cost it
// about 0.7 cycles each.  n = 1,048,576, m = 256: 243 ms, from 441 ms with the
// selection tested per step in FP64 and the bands in order of length (one gate per
// pass and 5 operations: 254 ms; that with a pass's two chunks as a loop 271 ms;
// 3 CTAs of 4 warps per SM at 168 registers spill, 273 ms).  Short windows have rows
// of unlike best scores side by side, and one bound for a pass's 23 rows and 16
// columns opened a quarter of the passes at m = 64 where 2% select (n = 600,000: 164
// ms; a bound per 15 rows and 8 columns 134; per 8 rows and a column 101, 97 with the passes
// after an open one straight).  With
// fewer bands than resident warps the longest band sets the time; then the bands
// are cut into tiles (Fp64Split).
#include <float.h>
#include <limits.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_prep_device.cuh"

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
// Scale and mean term of a record.
__device__ __forceinline__ double2 scale_mean(const double4* rec) {
    return __ldg(reinterpret_cast<const double2*>(rec) + 1);
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

// A row's best cell of the band: merged into its key slot.
__device__ __forceinline__ void flush_row(const Fp64BandParams& P, int shard, int64_t r, double score,
                                          int j) {
    if (score > P.floor) flush_fp64(P, shard, r + P.row_key_off, score, j + P.col_nb_off);
}
// Row t of tile lt (its rows start at rb; seg > 0: the band has a tile before it;
// more: one after it) has met the whole tile.
template <int R>
__host__ __device__ __forceinline__ bool seam_row(int64_t t, int64_t L, int64_t seg, bool more) {
    return (seg > 0 && t < 32 * R) || (more && t >= L);
}
template <int R, bool WHOLE>
__device__ __forceinline__ void finish_row(const Fp64BandParams& P, int shard, int64_t lt, int64_t seg,
                                           bool more, int64_t rb, int64_t t, double score, int j) {
    if (!WHOLE && seam_row<R>(t, P.split.L, seg, more)) {
        const int64_t i = lt * fp64_seam_rows(P.split.L, 32 * R) + fp64_seam_slot(t, P.split.L, 32 * R);
        P.split.seam_s[i] = score;
        P.split.seam_j[i] = j;
    } else if (j >= 0) {
        flush_row(P, shard, rb + t, score, j);
    }
}

// One warp's shared memory.  Rows of the band go in groups of R (row t of the
// tile, counted from its first column's row on the band's first diagonal, is
// element t % R of group t / R); kGroups slots of R rows form a ring, in which
// chunk c reads groups c .. c + 32; a pass of kU chunks copies in the next kU
// groups meanwhile.  Every
// array is padded by one element per group, so that lanes reading the same
// element of consecutive groups hit distinct banks (a multiple of 8 groups, so
// that a wrap keeps that for the 16-byte halves of the records).  A pass is 16
// columns for every R: half a warp brings in its columns, the other half its rows,
// and what a pass costs by itself is spread over as many columns (passes of 2R
// columns at R = 2, a block of 500 diagonals: the same 1.46 ms, but a pass's own
// instructions then weigh 4 times as much).
template <int R>
struct BandSmem {
    static constexpr int kU = 16 / R;  // chunks per pass
    static constexpr int kGroups = (32 + 2 * kU + 7) / 8 * 8;
    static_assert(kGroups % kU == 0 && kU * R <= kFp64SplitUnit, "tiles end with a pass");
    __device__ static __forceinline__ int wrap(int s) { return s < kGroups ? s : s - kGroups; }
    static constexpr int kRecStride = 32 * R + 16;  // bytes of a group's records
    static constexpr int kGateStride = R == 8 ? 12 : R;  // lanes hit distinct banks
    static constexpr int kUsed = kGroups * kRecStride + 2 * 32 * R * kU +
                                 kGroups * (R + 1) * (int)(sizeof(double) + sizeof(int)) +
                                 3 * R * kU * (int)sizeof(double) + R * kU * (int)sizeof(int) +
                                 (kGroups * kGateStride + 2 * R * kU + kGroups / kU) * (int)sizeof(int);
    static constexpr int kBytes = (kUsed + 15) / 16 * 16;  // warps' areas stay aligned
    char* rec;     // row records
    char* col;     // column records {A[j], A[j+m], s, fp64_gate_mean}, two buffers of kU * R
    double* best;  // best score of each row (fp64_bound of its threshold while src < 0)
    double* cmean; // column mean terms, two buffers of kU * R
    double* cbest; // best scores of the pass's columns ...
    int* cdiag;    // ... and their diagonals
    int* src;      // column of a row's best score, -1: none yet
    int* gate;     // per row: smallest gate among the best scores of R rows from it on
    int* cgate;    // gates of the columns' thresholds, two buffers of kU * R
    int* err;      // per kU groups: largest fp64_gate_error among the rows
    __device__ __forceinline__ BandSmem(char* p) {
        rec = p;
        p += kGroups * kRecStride;
        col = p;
        p += 2 * 32 * R * kU;
        best = reinterpret_cast<double*>(p);
        p += kGroups * (R + 1) * sizeof(double);
        cmean = reinterpret_cast<double*>(p);
        p += 2 * R * kU * sizeof(double);
        cbest = reinterpret_cast<double*>(p);
        p += R * kU * sizeof(double);
        src = reinterpret_cast<int*>(p);
        p += kGroups * (R + 1) * sizeof(int);
        gate = reinterpret_cast<int*>(p);
        cgate = gate + kGroups * kGateStride;
        err = cgate + 2 * R * kU;
        cdiag = err + kGroups / kU;
    }
    // gates of the rows of the group in slot s, from the best scores as they stand
    __device__ __forceinline__ void group_gates(int s, double m) const {
        const double *b0 = best + s * (R + 1), *b1 = best + wrap(s + 1) * (R + 1);
        const int hmin = fp64_gate_high_from(m);
        int x[2 * R - 1], run = INT_MIN;
#pragma unroll
        for (int k = 0; k < 2 * R - 1; ++k)
            x[k] = fp64_gate_high(__double2hiint(k < R ? b0[k] : b1[k - R]), hmin);
#pragma unroll
        for (int k = R - 2; k >= 0; --k) x[k] = max(x[k], x[k + 1]);
        int* g = gate + s * kGateStride;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (k > 0) run = max(run, x[R - 1 + k]);
            g[k] = max(x[k], run);
        }
    }
};

// The column's best cell over the warp, from two REDUX instructions (high, then
// low word of the ordered score; ties go to the smallest diagonal), left for the pass's
// end, which merges its 16 columns side by side (one lane's merge after each column took
// 107 of 274 ms where three of five columns select).  Returns whether there is one.
template <int R>
__device__ __forceinline__ bool select_column(const double (&sc)[R], double floor, double* best, int* diag,
                                              int lane) {
    // lane's best cell of the column.  A NaN cell (a constant window) never
    // selects under the reference's '>'; as -DBL_MAX it also cannot hide the
    // cell it is paired with in the tree.
    double cb[R];
#pragma unroll
    for (int a = 0; a < R; ++a) cb[a] = sc[a] == sc[a] ? sc[a] : -DBL_MAX;
#pragma unroll
    for (int w = 1; w < R; w *= 2)
#pragma unroll
        for (int a = 0; a + w < R; a += 2 * w) cb[a] = cb[a + w] > cb[a] ? cb[a + w] : cb[a];
    const double cbest = cb[0];
    const unsigned long long key = (cbest > floor) ? ord_f64(cbest) : 0ull;
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(kFullMask, hi);
    const unsigned mlo = __reduce_max_sync(kFullMask, hi == mhi ? lo : 0u);
    const bool top = (hi == mhi) && (lo == mlo) && (mhi != 0u);
    const unsigned tops = __ballot_sync(kFullMask, top);
    if (top && (tops & ((1u << lane) - 1u)) == 0u) {
        int ca = R - 1;
#pragma unroll
        for (int a = R - 2; a >= 0; --a) ca = sc[a] == cbest ? a : ca;
        *best = cbest;
        *diag = lane * R + ca;
    }
    return tops != 0u;
}

// A column step's selection: every cell above its row's best replaces it (strict '>', the
// reference's rule; a step's cells lie in distinct rows), and where some lane's cells may
// exceed the column's threshold (`col`) the column is reduced over the warp.  Cell a lies
// in element k + a of the lane's groups, which start at e0 and e1 + R; b: the column in
// the pass.  Returns kRose if a row's best rose in the lane, and bit b if the column has a
// best cell.
constexpr int kRose = 1 << 16;
template <int R>
struct Cells {
    double s[R];
};
template <int R>
__device__ __forceinline__ int select_cells(const Cells<R>& sc, double floor, unsigned j, const BandSmem<R>& sm,
                                            int e0, int e1, int k, int b, bool col, int lane) {
    __syncwarp();  // rows move from lane to lane between steps
    int did = 0;
    double best[R];
#pragma unroll
    for (int a = 0; a < R; ++a) best[a] = sm.best[(k + a < R ? e0 : e1) + a];
#pragma unroll
    for (int a = 0; a < R; ++a)
        if (sc.s[a] > best[a]) {
            sm.best[(k + a < R ? e0 : e1) + a] = sc.s[a];
            sm.src[(k + a < R ? e0 : e1) + a] = (int)j;
            did = kRose;
        }
    if (__any_sync(kFullMask, col) && select_column<R>(sc.s, floor, sm.cbest + b, sm.cdiag + b, lane))
        did |= 1 << b;
    return did;
}

// One chunk = R consecutive columns, all their cells in the reference's 4-wide
// (fused) part, without the selection: the largest high word of the lane's
// scores.  On entry rwin holds the records of the lane's first group (slot s1 - 1),
// on return those of its second.
template <int R>
__device__ __forceinline__ int gate_chunk(const BandSmem<R>& sm, int s0, int s1, const char* col,
                                          const int* cgate, double4 (&rwin)[R], double (&qt)[R]) {
    int over = INT_MIN;
    const int* gate = sm.gate + s0 * BandSmem<R>::kGateStride;
    const char* rec1 = sm.rec + s1 * BandSmem<R>::kRecStride;
    double4 cv = ring_rec(col);
#pragma unroll
    for (int b = 0; b < R; ++b) {
        double4 cn = cv;
        if (b + 1 < R) cn = ring_rec(col + 32 * (b + 1));
        double sc[R];
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const double4 rv = rwin[(b + a) % R];
            // the window moves on: element b + R replaces element b
            if (a == 0) rwin[b] = ring_rec(rec1 + 32 * b);
            // score / s of the column; the running dot product is the reference's
            // (kernels.cpp:206-225)
            sc[a] = __fma_rn(-rv.w, cv.w, __dmul_rn(rv.z, qt[a]));
            qt[a] = __fma_rn(-rv.x, cv.x, __fma_rn(rv.y, cv.y, qt[a]));
        }
        int top = 0;
        if (R == 1) top = max(top, __double2hiint(sc[0]));
#pragma unroll
        for (int a = 0; a + 1 < R; a += 2)
            top = __vimax3_s32(top, __double2hiint(sc[a]), __double2hiint(sc[a + 1]));
        top = fp64_gate_value(top, cv.z);
        cv = cn;
        over = __viaddmax_s32(top, gate[b], over);
        over = __viaddmax_s32(top, cgate[b], over);
    }
    return over;
}

// Whether a lane's pass with errors above the gates' slack opens (`over`: its largest
// value over its gate).
template <int R>
__device__ __noinline__ int widen_gate(const BandSmem<R>& sm, int s0, const int* cgate, int err,
                                       int over) {
    constexpr int kU = BandSmem<R>::kU;
    int g = cgate[0];
#pragma unroll
    for (int b = 1; b < kU * R; ++b) g = max(g, cgate[b]);
#pragma unroll
    for (int u = 0; u < kU; ++u)  // each covers R rows from its own on
        g = max(g, sm.gate[BandSmem<R>::wrap(s0 + u) * BandSmem<R>::kGateStride]);
    g = max(g, sm.gate[BandSmem<R>::wrap(s0 + kU - 1) * BandSmem<R>::kGateStride + R - 1]);
    return fp64_gate_lowered(g, err, over) ? 0 : -1;
}

// The same with the reference's arithmetic, a test of C columns at a time against the rows'
// own best scores: stops before the first C that hold a cell which may select.  Returns
// that column, R if there is none.
template <int R>
__device__ __forceinline__ int test_chunk(const BandSmem<R>& sm, int s0, int s1, const char* col,
                                          const double* cmean, const int* cgate, double4 (&rwin)[R],
                                          int (&gwin)[R], double (&qt)[R]) {
    const char* rec1 = sm.rec + s1 * BandSmem<R>::kRecStride;
    const double* best1 = sm.best + s1 * (R + 1);
    constexpr int C = R < 4 ? R : 4;
#pragma unroll
    for (int b0 = 0; b0 < R; b0 += C) {
        int over = INT_MIN;
        double q[R];
#pragma unroll
        for (int a = 0; a < R; ++a) q[a] = qt[a];
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int b = b0 + i;
            const double4 cv = ring_rec(col + 32 * b);
            const double cw = cmean[b];
            int top = 0, hi[R], o[2] = {INT_MIN, INT_MIN};
#pragma unroll
            for (int a = 0; a < R; ++a) {
                const double4 rv = rwin[(b + a) % R];
                const int rg = gwin[(b + a) % R];
                if (a == 0) {
                    rwin[b] = ring_rec(rec1 + 32 * b);
                    gwin[b] = fp64_best_gate(__double2hiint(best1[b]));
                }
                // kernels.cpp:206-225
                const double mm = __dmul_rn(cw, rv.w);
                const double sc = __fma_rn(q[a], __dmul_rn(rv.z, cv.z), -mm);
                q[a] = __fma_rn(-rv.x, cv.x, __fma_rn(rv.y, cv.y, q[a]));
                hi[a] = fp64_cell_high(__double2hiint(sc));
                o[a & 1] = __viaddmax_s32(hi[a], rg, o[a & 1]);
            }
            if (R == 1) top = hi[0];
#pragma unroll
            for (int a = 0; a + 1 < R; a += 2) top = __vimax3_s32(top, hi[a], hi[a + 1]);
            over = __vimax3_s32(over, o[0], o[1]);
            over = __viaddmax_s32(top, fp64_cell_gate(cgate[b]), over);
        }
        if (__any_sync(kFullMask, over >= kFp64Pass)) return b0;
#pragma unroll
        for (int a = 0; a < R; ++a) qt[a] = q[a];
    }
    return R;
}

// Columns `from` to `to` of a pass with the selection, s0 the slot of the lane's first
// group: EDGE evaluates every cell with its own geometry and selects in every step;
// otherwise all cells are fused and a step selects behind the gate.  Returns the steps'
// select_cells.  One loop over the columns with the records read from shared memory:
// unrolled like gate_chunk, this path's code pushed the passes without selection out of
// the instruction cache.
template <int R, bool EDGE>
__device__ __forceinline__ int select_pass(const Fp64BandParams& P, unsigned jc, const BandSmem<R>& sm, int s0,
                                           const char* col, const double* cmean, const int* cgate,
                                           double (&qt)[R], unsigned geo, int64_t gb, int lane, int from, int to) {
    constexpr int RS = BandSmem<R>::kRecStride;
    int did = 0;
#pragma unroll 1
    for (int b = from; b < to; ++b) {
        const unsigned j = jc + b;
        const int k = b % R;  // cell a lies in element k + a of the lane's groups
        const int sa = BandSmem<R>::wrap(s0 + b / R), sb = BandSmem<R>::wrap(sa + 1);
        const char* rec0 = sm.rec + sa * RS + 32 * k;
        const char* rec1 = sm.rec + sb * RS + 32 * (k - R);
        const double4 cv = ring_rec(col + 32 * b);
        const double cw = cmean[b];
        Cells<R> sc;
        int top = kFp64NoNan;
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const double4 rv = ring_rec((k + a < R ? rec0 : rec1) + 32 * a);
            double score = -DBL_MAX;
            const unsigned code = (geo >> (4 * a)) & 15u;
            const int64_t left = P.Tbase - gb - (lane * R + a) - (int64_t)j;  // columns from j on
            if (!EDGE || (code != 15u && left > 0)) {
                const double ss = __dmul_rn(rv.z, cv.z);
                if (!EDGE || (code != 7u && left >= 4 - (int)code)) {
                    // kernels.cpp:206-225
                    const double mm = __dmul_rn(cw, rv.w);
                    score = __fma_rn(qt[a], ss, -mm);
                    qt[a] = __fma_rn(-rv.x, cv.x, __fma_rn(rv.y, cv.y, qt[a]));
                } else {
                    // scalar remainder (kernels.cpp:282-289), no fusion
                    score = __dsub_rn(__dmul_rn(qt[a], ss), __dmul_rn(rv.w, cw));
                    qt[a] = __dsub_rn(__dadd_rn(qt[a], __dmul_rn(rv.y, cv.y)),
                                      __dmul_rn(rv.x, cv.x));
                }
            }
            sc.s[a] = score;
            top = __viaddmax_s32(__double2hiint(score), kFp64NoNan, top);
        }
        top -= kFp64NoNan;
        if (!EDGE &&
            !__any_sync(kFullMask, top + max(sm.gate[sa * BandSmem<R>::kGateStride + k], cgate[b]) >= 0))
            continue;
        did |= select_cells<R>(sc, P.floor, j, sm, sa * (R + 1) + k, sb * (R + 1) + k - R, k, b,
                               top + cgate[b] >= 0, lane);
    }
    return did;
}

// Columns [j0, jend) of a band.  lt: the tile's number when the band is cut into
// tiles (then jend - j0 = L, or less for the band's last tile).  WHOLE: see above.
template <int R, bool WHOLE>
__device__ __forceinline__ void band_fp64(const Fp64BandParams& P, int64_t band, int64_t lt,
                                          int64_t seg, int lane, int shard,
                                          const BandSmem<R>& sm) {
    constexpr int RS = BandSmem<R>::kRecStride, kU = BandSmem<R>::kU, kGroups = BandSmem<R>::kGroups;
    const int64_t gb = P.g_lo + band * (int64_t)(32 * R);
    const int64_t g0 = gb + (int64_t)lane * R;
    const int64_t jmax = P.Tbase - gb;  // length of the band's longest diagonal
    const int64_t L = P.split.L;
    const unsigned j0 = (unsigned)(seg * L);
    if ((int64_t)j0 >= jmax) return;
    const bool more = !WHOLE && L > 0 && j0 + L < jmax;  // the band goes on in the next tile
    const unsigned jend = more ? j0 + (unsigned)L : (unsigned)jmax;
    const int64_t rb = gb + j0;  // row t = 0 of the tile

    // Diagonal g has len = Tbase - g columns; with delta its offset in its block,
    // its last column of the reference's 4-wide part is len - 4 + delta % 4, or
    // none when delta >= B & ~3.  geo holds delta % 4 (or 7) of the lane's
    // diagonals, 15 for one past g_hi, as nibbles: only the chunks near a
    // diagonal's end read them.  A diagonal past g_hi, or one that ended before
    // the tile, carries -inf, which stays below every bound, so it does not cost
    // the tile its branch-free passes.
    double qt[R];
    unsigned geo = 0;
    int minpsw = INT_MAX;
    int64_t delta = (g0 - P.blk_origin) % P.B;
#pragma unroll
    for (int a = 0; a < R; ++a) {
        const int64_t g = g0 + a;
        unsigned code = 15;
        qt[a] = -__longlong_as_double(0x7ff0000000000000ll);
        if (g < P.g_hi && (int64_t)j0 < P.Tbase - g) {
            qt[a] = seg == 0 ? P.qt0[g - P.g_lo]
                             : P.split.seeds[(seg - 1) * (P.g_hi - P.g_lo) + (g - P.g_lo)];
            code = delta < (P.B & ~3ll) ? (unsigned)(delta & 3) : 7u;
            minpsw = min(minpsw, code == 7u ? -1 : (int)(P.Tbase - g) - 4 + (int)code);
        }
        geo |= code << (4 * a);
        delta = delta + 1 == P.B ? 0 : delta + 1;
    }
    minpsw = __reduce_min_sync(kFullMask, minpsw);

    // Groups 0 .. 32 + kU - 1 and the first pass's columns.  In a pass, lanes R to
    // R + 15 bring in what belongs to the next 16 rows, the others to the next 16
    // columns; part: which one.
    static_assert(kU * R == 16, "half a warp each");
    const bool isrow = lane >= R && lane < R + 16;
    const int part = isrow ? lane - R : lane & 15;
    const uint4* rsrc = reinterpret_cast<const uint4*>(P.rowrec + rb);
    const uint4* crec = reinterpret_cast<const uint4*>(P.colrec + j0);
    const double* tsrc = P.thr + rb + P.row_key_off;  // threshold of row t
    const double* csrc = P.thr + j0 + P.col_key_off;  // threshold of column j0
    const int64_t wlast = P.Tbase - 1;                // colgate ends there
    const int errfree = fp64_gate_errfree(P.m);
    for (int i = lane; i < (32 + kU) * 2 * R; i += 32)
        cp_async16(sm.rec + (i / (2 * R)) * RS + 16 * (i % (2 * R)), rsrc + i);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    constexpr int kOwn = (32 * R + 16 + 31) / 32;  // rows that a lane brings in
    double thr[kOwn];
    double2 sw[kOwn];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {  // all in flight together (the last ones may be past the tile's)
        thr[k] = ld_thr(tsrc + lane + 32 * k);
        sw[k] = scale_mean(P.rowrec + rb + lane + 32 * k);
    }
    int rerr = 0;  // one bound for all rows that the tile starts with
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        const int i = lane + 32 * k;
        if (i < (32 + kU) * R) {
            sm.best[(i / R) * (R + 1) + i % R] = fp64_bound(thr[k], sw[k].x, sw[k].y);
            sm.src[(i / R) * (R + 1) + i % R] = -1;
            rerr = max(rerr, fp64_gate_error(sw[k].x, sw[k].y));
        }
    }
    rerr = __reduce_max_sync(kFullMask, rerr);
    int cerr = 0;
    if (lane < R * kU) {
        const double t = ld_thr(csrc + lane);
        const double2 sw = scale_mean(P.colrec + j0 + lane);
        *reinterpret_cast<uint4*>(sm.col + 32 * lane) = __ldg(crec + 2 * lane);
        *reinterpret_cast<double2*>(sm.col + 32 * lane + 16) =
            make_double2(sw.x, __ldg(P.colgate + min((int64_t)j0 + lane, wlast)));
        sm.cmean[lane] = sw.y;
        sm.cgate[lane] = fp64_gate(fp64_bound(t, sw.x, sw.y), P.m);
        cerr = fp64_gate_error(sw.x, sw.y);
    }
    cerr = __reduce_max_sync(kFullMask, cerr);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    for (int s = lane; s + 1 < 32 + kU; s += 32) sm.group_gates(s, P.m);
    if (lane < kGroups / kU) sm.err[lane] = rerr;
    // lanes 0 to R - 1: gates of the last group brought in
    int lastg = fp64_gate(sm.best[(32 + kU - 1) * (R + 1) + lane % R], P.m);
    __syncwarp();
    // register window of row records: slot (k mod R) holds element k of the
    // lane's first group
    double4 rwin[R];
    auto load_window = [&](int s) {
#pragma unroll
        for (int k = 0; k < R; ++k) rwin[k] = ring_rec(sm.rec + s * RS + 32 * k);
    };
    load_window(lane);

    // what the lane copies in next: records of groups c + 32 + kU .. and of the
    // next pass's columns, and their thresholds
    const uint4* nrow = rsrc + (32 + kU) * 2 * R + lane;
    const double* nthr = isrow ? tsrc + (32 + kU) * R + part : csrc + kU * R + part;
    const double4* nrec = isrow ? P.rowrec + rb + (32 + kU) * R + part : P.colrec + j0 + kU * R + part;
    int64_t nw = (int64_t)j0 + kU * R + part;  // its index in colgate (columns)
    int s0 = lane;  // slot of the lane's first group
    int sf = 0;     // slot of group c, the first that the pass finishes
    int cbuf = 0;
    bool sel = false;
    int skip = 0, streak = 0;
    for (unsigned jc = j0; jc < jend; jc += kU * R) {
        const int sn = BandSmem<R>::wrap(sf + 32 + kU);  // slots of the incoming groups (kU divides kGroups)
        double w = 0.0;
        cp_async16(sm.rec + (sn + lane / (2 * R)) * RS + 16 * (lane % (2 * R)), nrow);
        const double t = ld_thr(nthr);
        const double2 sw = scale_mean(nrec);
        if (!isrow) {
            w = __ldg(P.colgate + min(nw, wlast));
            cp_async16(sm.col + (cbuf ^ 1) * (32 * R * kU) + 32 * part, nrec);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        nrow += kU * 2 * R;
        nthr += kU * R;
        nrec += kU * R;
        nw += kU * R;
        const char* col = sm.col + cbuf * (32 * R * kU);
        const int* cgate = sm.cgate + cbuf * (R * kU);
        const double* cmean = sm.cmean + cbuf * (R * kU);
        const bool fused = (int64_t)jc + (kU * R - 1) <= minpsw;
        // A pass after one that selected goes straight to selecting; so do the next 1, 2,
        // 4 .. 16 passes after gates that opened in a row.
        bool open = !fused || sel || skip > 0;
        skip -= skip > 0;
        if (!open) {
            double q0[R];
#pragma unroll
            for (int a = 0; a < R; ++a) q0[a] = qt[a];
            int over = INT_MIN;
            const int err = max(cerr, max(sm.err[s0 / kU], sm.err[BandSmem<R>::wrap(s0 + kU) / kU]));
#pragma unroll
            for (int u = 0; u < kU; ++u)
                over = max(over, gate_chunk<R>(sm, BandSmem<R>::wrap(s0 + u), BandSmem<R>::wrap(s0 + u + 1),
                                               col + u * 32 * R, cgate + u * R, rwin, qt));
            if (err > errfree) over = widen_gate<R>(sm, s0, cgate, err, over);
            open = __any_sync(kFullMask, over >= 0);
            streak = WHOLE && open ? min(max(2 * streak, 1), 16) : 0;
            skip = streak;
            if (open) {
#pragma unroll
                for (int a = 0; a < R; ++a) qt[a] = q0[a];
                if (WHOLE) load_window(s0);
            }
        }
        sel = false;
        int did = 0;
        if (open && !(WHOLE && fused)) {
            did = fused ? select_pass<R, false>(P, jc, sm, s0, col, cmean, cgate, qt, geo, gb, lane, 0, kU * R)
                        : select_pass<R, true>(P, jc, sm, s0, col, cmean, cgate, qt, geo, gb, lane, 0, kU * R);
            load_window(BandSmem<R>::wrap(s0 + kU));
        } else if (open) {
#pragma unroll 1
            for (int u = 0; u < kU; ++u) {
                const int sa = BandSmem<R>::wrap(s0 + u), sb = BandSmem<R>::wrap(sa + 1);
                int gwin[R];  // gates of the rows in rwin
#pragma unroll
                for (int a = 0; a < R; ++a) gwin[a] = fp64_best_gate(__double2hiint(sm.best[sa * (R + 1) + a]));
                const int b = test_chunk<R>(sm, sa, sb, col + u * 32 * R, cmean + u * R, cgate + u * R, rwin,
                                            gwin, qt);
                if (b < R) {
                    did |= select_pass<R, false>(P, jc, sm, s0, col, cmean, cgate, qt, geo, gb, lane, u * R + b,
                                                 (u + 1) * R);
                    load_window(sb);
                }
            }
        }
        if (open) {
            sel = __any_sync(kFullMask, did & kRose);
            __syncwarp();
            if ((did & (kRose - 1)) >> lane & 1) {  // column jc + lane
                const int64_t j = (int64_t)jc + lane;
                flush_fp64(P, shard, j + P.col_key_off, sm.cbest[lane], j + gb + sm.cdiag[lane] + P.row_nb_off);
            }
        }
        __syncwarp();
        // groups c .. c + kU - 1 have met every lane: merge their rows
        if (lane < R * kU) {
            const int e = (sf + lane / R) * (R + 1) + lane % R;
            const int j = sm.src[e];
            finish_row<R, WHOLE>(P, shard, lt, seg, more, rb, (int64_t)(jc - j0) + lane, sm.best[e], j);
        }
        // the incoming groups and columns begin at their thresholds
        const double bound = fp64_bound(t, sw.x, sw.y);
        const int x = fp64_gate(bound, P.m);
        if (isrow) {
            const int e = (sn + part / R) * (R + 1) + part % R;
            sm.best[e] = bound;
            sm.src[e] = -1;
        } else {
            *reinterpret_cast<double2*>(sm.col + (cbuf ^ 1) * (32 * R * kU) + 32 * part + 16) =
                make_double2(sw.x, w);
            sm.cmean[(cbuf ^ 1) * (R * kU) + part] = sw.y;
            sm.cgate[(cbuf ^ 1) * (R * kU) + part] = x;
        }
        // one bound of the errors for the rows and the columns
        cerr = __reduce_max_sync(kFullMask, fp64_gate_error(sw.x, sw.y));
        if (lane == 0) sm.err[sn / kU] = cerr;
        // gates of the last incoming group of the pass before (its rows' minima reach
        // into this one's) and of all but the last of this one's: its rows are in
        // lanes 0 to R - 1, this one's follow
        int win = lane < R ? lastg : isrow ? x : INT_MIN;
#pragma unroll
        for (int d = 1; d < R; d *= 2) win = max(win, __shfl_down_sync(kFullMask, win, d));
        if (lane < kU * R) {
            const int s = lane < R ? (sn == 0 ? kGroups : sn) - 1 : sn + lane / R - 1;
            sm.gate[s * BandSmem<R>::kGateStride + lane % R] = win;
        }
        lastg = __shfl_sync(kFullMask, x, (lane + 16) & 31);
        s0 = BandSmem<R>::wrap(s0 + kU);
        if (sel) {  // best scores of groups c + kU .. c + kU + 31 rose
            __syncwarp();
            sm.group_gates(s0, P.m);
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        sf = BandSmem<R>::wrap(sf + kU);
        cbuf ^= 1;
    }

    // drain: rows of groups c .. c + 31 (the last chunk's second groups)
    const int64_t tend = ((int64_t)(jend - j0) + kU * R - 1) / (kU * R) * (kU * R);  // row t of group c
    for (int i = lane; i < 32 * R; i += 32) {
        const int e = BandSmem<R>::wrap(sf + i / R) * (R + 1) + i % R;
        const int j = sm.src[e];
        finish_row<R, WHOLE>(P, shard, lt, seg, more, rb, tend + i, sm.best[e], j);
    }
    __syncwarp();

    if (P.qt_out) {  // diagonals whose last column lies in the tile
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const int64_t g = g0 + a, len = P.Tbase - g;
            if (g < P.g_hi && (int64_t)j0 < len && len <= (int64_t)jend) P.qt_out[g - P.g_lo] = qt[a];
        }
    }
}

template <int R>
constexpr int fp64_smem_bytes() {
    return kFp64WarpsPerBlock * BandSmem<R>::kBytes;
}

template <int R, bool WHOLE>
__global__ void __launch_bounds__(32 * kFp64WarpsPerBlock, R == 8 ? 2 : 4)
    fp64_band_kernel(const Fp64BandParams P) {
    extern __shared__ __align__(128) char smem_fp64[];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const BandSmem<R> sm(smem_fp64 + w * BandSmem<R>::kBytes);
    // One resident wave of W warps takes the bands by rank (fp64_band_of), or the
    // tiles by number: warp w starts with rank w, later ranks come from one
    // counter (no waiting on anything).
    const int64_t wid = (int64_t)blockIdx.x * kFp64WarpsPerBlock + w;
    const int shard = (int)(wid % P.shards);
    const int64_t count = P.split.L > 0 ? P.split.ntiles : P.nbands;
    for (int64_t rank = wid; rank < count;) {
        int64_t band, seg = 0;
        bool any = true;
        if (P.split.L > 0)
            any = tile_of_pair(rank, P.Tbase, P.g_lo, P.split.L, P.nbands, P.split.seg_per_pair,
                               32 * R, band, seg);
        else
            band = fp64_band_of(rank, P.nbands, P.spread);
        if (any) band_fp64<R, WHOLE>(P, band, rank, seg, lane, shard, sm);
        unsigned next = 0;
        if (lane == 0) next = atomicAdd(P.counter, 1u);
        rank = (int64_t)gridDim.x * kFp64WarpsPerBlock + __shfl_sync(kFullMask, next, 0);
    }
}

// Rows met by several tiles of a band: the block of tile lt takes the rows whose
// last tile (or the band's last) it is; the earlier tile's cell (smaller column)
// wins ties, as within a tile.
template <int R>
__global__ void fp64_seam_kernel(const Fp64BandParams P) {
    const int64_t lt = blockIdx.x, L = P.split.L, stride = L + 32 * R;  // rows of a tile
    const int64_t slots = fp64_seam_rows(L, 32 * R);
    int64_t band, seg;
    if (!tile_of_pair(lt, P.Tbase, P.g_lo, L, P.nbands, P.split.seg_per_pair, 32 * R, band, seg) ||
        seg == 0)
        return;
    const int64_t gb = P.g_lo + band * (32 * R);
    const int64_t last = (P.Tbase - gb + L - 1) / L - 1;  // the band's last tile
    // rows x = t + seg L of the band: t < L, or all of the last tile's
    const int64_t rows = min((int64_t)(32 * R), seg == last ? stride : L);
    for (int64_t t = threadIdx.x; t < rows; t += blockDim.x) {
        const int64_t x = seg * L + t;
        double s = 0.0;
        int j = -1;
        for (int64_t k = max((int64_t)0, (x - stride) / L); k <= seg; ++k) {
            const int64_t tk = x - k * L;
            if (tk >= stride || !seam_row<R>(tk, L, k, k < last)) continue;
            const int64_t i = (lt - (seg - k)) * slots + fp64_seam_slot(tk, L, 32 * R);
            const int jk = P.split.seam_j[i];
            if (jk >= 0 && (j < 0 || P.split.seam_s[i] > s)) {
                s = P.split.seam_s[i];
                j = jk;
            }
        }
        if (j >= 0) flush_row(P, (int)(lt % P.shards), gb + x, s, j);
    }
}

// ---- running dot products at the tiles' first columns ------------------------
// The recurrence of a diagonal is a chain of two dependent FP64 operations per
// column, 8 cycles each, and a thread per diagonal cannot run ahead of it: 16
// cycles per column of the longest diagonal bound this kernel (n = 16,384: 0.14
// ms, 0.28 measured; n = 65,536: 0.55 ms, 1.10 measured).  Above two blocks of
// diagonals per SM a thread walks C = 4 adjacent ones, so that 4 chains overlap
// and a value of the series read from shared memory serves 4.  Operands are
// staged there a chunk ahead; row values lie C + 1 apart per C, so that lanes hit
// distinct banks.  The series' prefix sums, which only the join needs, are another
// serial chain and run beside the seeds in one more block (n = 65,536: 3.13 -> 2.78
// ms per call; n = 2,500: 194 -> 184 us).
constexpr int kSeedThreads = 128;
constexpr int kSeedChunk = 128;
constexpr int kSeedPrefixChunk = 192;

template <int C>
__global__ void __launch_bounds__(kSeedThreads)
    fp64_seed_kernel(const Fp64BandParams P, const double* __restrict__ Ah, int64_t nh,
                     const double* __restrict__ Av, int64_t nv, int64_t m, const PrefixSums X) {
    constexpr int K = kSeedChunk, T = kSeedThreads;
    static_assert(K == T && T % 8 == 0 && (C == 1 || C == 4), "a thread stages one row and one column per chunk");
    // Ring of rows in blocks of K: a chunk reads rows [0, T*C + K) from its first
    // while the next K arrive; block 0 is mirrored behind the ring (with 8 + C
    // rows more, read ahead and not used), so a lane's rows of a chunk never wrap.
    constexpr int kBlocks = C + 2;
    constexpr int kRing = kBlocks * K + K + 16;
    constexpr int kPad = C > 1 ? kRing / C : 0;
    constexpr int kColBytes = 2 * (K + 16) * (int)sizeof(double2);
    constexpr int kBytes = kColBytes + 2 * (kRing + kPad) * (int)sizeof(double);
    static_assert(PrefixSmem<kSeedPrefixChunk>::kBytes <= kBytes, "the prefix block's buffers fit");
    __shared__ __align__(16) char smem[kBytes];
    if (X.n > 0 && blockIdx.x == 0) {
        prefix_block<kSeedPrefixChunk>(X.A, X.n, X.cs, X.cs2, smem);
        return;
    }
    auto scol = reinterpret_cast<double2(*)[K + 16]>(smem);                      // {A[j], A[j+m]}
    auto srow = reinterpret_cast<double(*)[kRing + kPad]>(smem + kColBytes);     // A[r], A[r+m]
    const int tid = threadIdx.x;
    const int64_t d0 = (int64_t)(blockIdx.x - (X.n > 0)) * (T * C);  // first diagonal, from g_lo
    const int64_t nd = P.g_hi - P.g_lo, L = P.split.L;
    const int64_t gb = P.g_lo + d0, g0 = gb + (int64_t)tid * C;
    const int64_t jlast = (P.Tbase - gb - 1) / L * L;     // start of the longest diagonal's last tile
    if (jlast <= 0) return;
    double q[C];
    int64_t psw[C], minpsw = P.Tbase;
#pragma unroll
    for (int a = 0; a < C; ++a) {
        const int64_t g = g0 + a;
        q[a] = 0.0;
        psw[a] = P.Tbase;
        if (g < P.g_hi) {
            const int64_t delta = (g - P.blk_origin) % P.B;
            q[a] = P.qt0[g - P.g_lo];
            psw[a] = delta < (P.B & ~3ll) ? P.Tbase - g - 4 + (delta & 3) : -1;
            // cells past a diagonal's last tile start feed nothing
            if (P.Tbase - g > L) minpsw = min(minpsw, psw[a]);
        }
    }
    // rows gb + i, i in block bi of the ring (i = K * (number of blocks before))
    auto stage_rows = [&](int64_t i, int bi) {
        const int64_t r = gb + i + tid;
        const bool in0 = r < nv, in1 = r + m < nv;
        const double *p0 = Av + (in0 ? r : 0), *p1 = Av + (in1 ? r + m : 0);
        int e = bi * K + tid;
        e += C > 1 ? e / C : 0;
        cp_async8_or_zero(&srow[0][e], p0, in0);
        cp_async8_or_zero(&srow[1][e], p1, in1);
        if (bi == 0) {
            e += kBlocks * K + (C > 1 ? kBlocks * K / C : 0);
            cp_async8_or_zero(&srow[0][e], p0, in0);
            cp_async8_or_zero(&srow[1][e], p1, in1);
        }
    };
    auto stage_cols = [&](int64_t jc, int buf) {
        const int64_t j = jc + tid;
        const bool in0 = j < nh, in1 = j + m < nh;
        cp_async8_or_zero(&scol[buf][tid].x, Ah + (in0 ? j : 0), in0);
        cp_async8_or_zero(&scol[buf][tid].y, Ah + (in1 ? j + m : 0), in1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int bi = 0; bi <= C; ++bi) stage_rows((int64_t)bi * K, bi);
    stage_cols(0, 0);
    // dot products at a tile's first column (kFp64SplitUnit columns apart or more)
    int64_t jnext = L;
    double* out = P.split.seeds + d0 + (int64_t)tid * C;
    auto leave = [&](int64_t j) {
        if (j != jnext) return;
#pragma unroll
        for (int a = 0; a < C; ++a)
            if (g0 + a < P.g_hi && j < P.Tbase - (g0 + a)) out[a] = q[a];
        jnext += L;
        out += nd;
    };
    int buf = 0;
    int bl = 0;  // block of the chunk's first row
    for (int64_t jc = 0;; jc += K, buf ^= 1, bl = bl + 1 == kBlocks ? 0 : bl + 1) {
        if (jc > jlast) break;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        // rows [T*C + K, T*C + 2K) from the chunk's first: the block before it
        stage_rows(jc + T * C + K, bl == 0 ? kBlocks - 1 : bl - 1);
        stage_cols(jc + K, buf ^ 1);
        // lane's first row of the chunk: block bl, element tid * C, modulo the ring
        int rs = bl * K + tid * C;
        rs = rs < kBlocks * K ? rs : rs - kBlocks * K;
        const double* ra = srow[0] + rs + (C > 1 ? rs / C : 0);
        const double* rm = srow[1] + rs + (C > 1 ? rs / C : 0);
        double wa[C], wm[C];  // rows of the current column: slot (column + a) % C
#pragma unroll
        for (int a = 0; a < C - 1; ++a) {
            wa[a] = ra[a];
            wm[a] = rm[a];
        }
        if (jc + K - 1 <= minpsw) {
            // The next U columns' operands are read into the other half of the
            // registers while these run, each read between the chain's dependent
            // operations.
            constexpr int U = 8;
            static_assert(K % (2 * U) == 0 && U % C == 0 && kFp64SplitUnit % (2 * U) == 0, "tiles start at a round");
            constexpr int kStep = C > 1 ? U + U / C : U;
            double xa[2][U], xm[2][U];
            double2 xc[2][U];
            auto fetch = [&](int h, int k, const double* pa, const double* pm, const double2* pc) {
                const int i = k + C - 1, e = C > 1 ? i + i / C : i;
                xa[h][k] = pa[e];
                xm[h][k] = pm[e];
                xc[h][k] = pc[k];
            };
            const double2* pc = scol[buf];
#pragma unroll
            for (int k = 0; k < U; ++k) fetch(0, k, ra, rm, pc);
            auto walk = [&](auto starts) {  // starts: a tile starts in the chunk
#pragma unroll 1
                for (int k0 = 0; k0 < K; k0 += 2 * U) {
                    if (decltype(starts)::value) leave(jc + k0);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        ra += kStep;
                        rm += kStep;
                        pc += U;
#pragma unroll
                        for (int k = 0; k < U; ++k) {
                            wa[(k + C - 1) % C] = xa[h][k];
                            wm[(k + C - 1) % C] = xm[h][k];
#pragma unroll
                            for (int a = 0; a < C; ++a) q[a] = __fma_rn(wm[(k + a) % C], xc[h][k].y, q[a]);
                            fetch(h ^ 1, k, ra, rm, pc);  // past the chunk: read, not used
#pragma unroll
                            for (int a = 0; a < C; ++a) q[a] = __fma_rn(-wa[(k + a) % C], xc[h][k].x, q[a]);
                        }
                    }
                }
            };
            if (jnext < jc + K)
                walk(std::true_type{});
            else
                walk(std::false_type{});
        } else {
#pragma unroll 1
            for (int k0 = 0; k0 < K; k0 += 4) {
                leave(jc + k0);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = k + C - 1, e = C > 1 ? i + i / C : i;
                    wa[i % C] = ra[e];
                    wm[i % C] = rm[e];
                    const double2 c = scol[buf][k0 + k];
#pragma unroll
                    for (int a = 0; a < C; ++a) {
                        const double x = wa[(k + a) % C], y = wm[(k + a) % C];
                        if (jc + k0 + k <= psw[a])
                            q[a] = __fma_rn(-x, c.x, __fma_rn(y, c.y, q[a]));
                        else  // the reference's scalar remainder
                            q[a] = __dsub_rn(__dadd_rn(q[a], __dmul_rn(y, c.y)), __dmul_rn(x, c.x));
                    }
                }
                ra += C > 1 ? 4 + 4 / C : 4;
                rm += C > 1 ? 4 + 4 / C : 4;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

}  // namespace

Fp64Split fp64_split_plan(int64_t Tbase, int64_t g_lo, int64_t g_hi, int R, size_t room) {
    Fp64Split S{};
    const int64_t span = 32 * R, nd = g_hi - g_lo;
    if (nd <= 0) return S;
    const int64_t nbands = (nd + span - 1) / span;
    // Whole bands keep the chip busy once there are about as many as resident
    // warps (8 per SM), and the dot products of the tiles' first columns cost two
    // more FP64 operations per cell.  Joins in tiles (with their seeds) against whole bands: n =
    // 2,500 0.08 / 0.81 ms; 16,384 0.6 / 2.2; 65,536 (256 bands) 2.3 / 6.4; 180,000 (702)
    // 12 / 16.4; 240,000 (936) 21 / 23.3; whole calls of 260,000 25.5 / 26.5, 300,000 33.5 / 31.3.
    const int64_t warps = (int64_t)sm_count() * 8;
    if (nbands > warps * 4 / 5) return S;
    // About 5 tiles per warp (10 and 20 measured the same; 2 per warp 16.8 ms at n =
    // 200,000, bands in 4 parts 16.4); at least 32 columns, for the smallest series,
    // whose tiles are all resident at once (n = 2,500: 32 columns 0.105 ms, 64 0.127,
    // 256 0.26).
    const int64_t cols = nbands * (Tbase - g_lo) - span * (nbands * (nbands - 1) / 2);
    int64_t L = std::max<int64_t>(cols / (5 * warps), 32);
    L = (L + kFp64SplitUnit - 1) / kFp64SplitUnit * kFp64SplitUnit;
    for (; L < Tbase - g_lo; L += (L / 2 + kFp64SplitUnit - 1) / kFp64SplitUnit * kFp64SplitUnit) {
        S.L = L;
        S.nseg = (Tbase - g_lo + L - 1) / L;
        int64_t nb = 0;
        fp32_tile_plan(Tbase, g_lo, g_hi, L, R, nb, S.seg_per_pair, S.ntiles);
        if (fp64_split_bytes(S, nd, R) <= room) return S;
    }
    return Fp64Split{};
}

size_t fp64_split_bytes(const Fp64Split& S, int64_t ndiag, int R) {
    if (S.L == 0) return 0;
    const size_t rows = (size_t)(S.ntiles * fp64_seam_rows(S.L, 32 * R));
    return align_up(8 * (size_t)((S.nseg - 1) * ndiag)) + align_up(8 * rows) + align_up(4 * rows);
}

void fp64_split_carve(Fp64Split& S, int64_t ndiag, int R, char* p) {
    S.seeds = reinterpret_cast<double*>(p);
    p += align_up(8 * (size_t)((S.nseg - 1) * ndiag));
    S.seam_s = reinterpret_cast<double*>(p);
    p += align_up(8 * (size_t)(S.ntiles * fp64_seam_rows(S.L, 32 * R)));
    S.seam_j = reinterpret_cast<int*>(p);
}

void launch_fp64_seeds(const Fp64BandParams& P, const double* Ah, int64_t nh, const double* Av,
                       int64_t nv, int64_t m, const PrefixSums& X, cudaStream_t s) {
    const unsigned more = X.n > 0;
    const int64_t nd = P.g_hi - P.g_lo;
    const int64_t blocks1 = (nd + kSeedThreads - 1) / kSeedThreads;
    if (blocks1 <= 2 * sm_count())
        fp64_seed_kernel<1><<<(unsigned)blocks1 + more, kSeedThreads, 0, s>>>(P, Ah, nh, Av, nv, m, X);
    else
        fp64_seed_kernel<4><<<(unsigned)((blocks1 + 3) / 4) + more, kSeedThreads, 0, s>>>(P, Ah, nh, Av, nv, m,
                                                                                    X);
}

template <int R, bool WHOLE>
void launch_band_kernel(const Fp64BandParams& Q, cudaStream_t s) {
    constexpr int smem = fp64_smem_bytes<R>();
    // per-device attribute and occupancy, idempotent: see launch_fp32_join
    static std::atomic<unsigned long long> configured{0};
    static std::atomic<int> resident[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(fp64_band_kernel<R, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fp64_band_kernel<R, WHOLE>,
                                                          32 * kFp64WarpsPerBlock, smem) != cudaSuccess ||
            per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        resident[dev & 63].store(per_sm, std::memory_order_relaxed);
        configured.fetch_or(bit, std::memory_order_release);
    }
    // one resident wave, fewer CTAs when there is less work than warps
    const int64_t wave = (int64_t)sm_count() * resident[dev & 63].load(std::memory_order_relaxed);
    const int64_t count = Q.split.L > 0 ? Q.split.ntiles : Q.nbands;
    const int64_t want = (count + kFp64WarpsPerBlock - 1) / kFp64WarpsPerBlock;
    const int64_t blocks = std::min<int64_t>(want, wave);
    if (blocks <= 0) return;
    Fp64BandParams P = Q;
    P.spread = (P.nbands + blocks * kFp64WarpsPerBlock - 1) / (blocks * kFp64WarpsPerBlock);
    cudaMemsetAsync(P.counter, 0, sizeof(unsigned), s);
    fp64_band_kernel<R, WHOLE><<<(unsigned)blocks, 32 * kFp64WarpsPerBlock, smem, s>>>(P);
    if (P.split.L > 0) fp64_seam_kernel<R><<<(unsigned)P.split.ntiles, 128, 0, s>>>(P);
}

// Whole bands of 256 diagonals take the kernel that backs off (m = 16, n = 280,000: 45 ms, 80
// without); narrower bands come from a few hundred diagonals, which are cut into tiles
// wherever there is room.
template <int R>
void launch_fp64_band(const Fp64BandParams& P, cudaStream_t s) {
    if (R == 8 && P.split.L == 0)
        launch_band_kernel<R, R == 8>(P, s);
    else
        launch_band_kernel<R, false>(P, s);
}

template void launch_fp64_band<1>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<2>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<4>(const Fp64BandParams&, cudaStream_t);
template void launch_fp64_band<8>(const Fp64BandParams&, cudaStream_t);

}  // namespace mpgpu
