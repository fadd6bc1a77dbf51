// Kernel declarations and launch parameter blocks shared by the mpgpu
// translation units (device code and the C-ABI layer).
#pragma once

#include <float.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstring>

struct mp_context;

namespace mpgpu {

// Memory budget of a context (0 = none); defined with the context in mp_capi.cu.
size_t ctx_budget(const mp_context* ctx);
int ctx_device(const mp_context* ctx);

// ---- preparation (mp_prep.cu) ----------------------------------------------
constexpr int kPrefixThreads = 256;  // ref_prefix_kernel: one block of this many threads
constexpr int kPrefixChunk = 736;    // elements of A per shared-memory chunk (48 KB of buffers)
__global__ void ref_prefix_kernel(const double* A, int64_t n, double* cs, double* cs2);
__global__ void ref_stats_kernel(const double* cs, const double* cs2, int64_t PL, int64_t m,
                                 double* muS, double* sInv);
__global__ void first_qt_kernel(const double* A, int64_t m, int64_t d_lo, int64_t d_hi,
                                double* qt);
__global__ void pack_fp64_kernel(const double* Apad, int64_t m, int64_t count, double* sInv,
                                 const double* muS, double4* rec);
__global__ void change_flags_kernel(const double* A, int64_t n, int* chg);
__global__ void scan_blocks_kernel(int* x, int64_t n, int* block_tot);
__global__ void scan_totals_kernel(int* tot, int64_t nblocks);
__global__ void scan_add_kernel(int* x, int64_t n, const int* tot);
__global__ void welford_kernel(const double* A, int64_t m, int64_t PL, int64_t chunk,
                               const int* nchg, double* mean_out, double* norm_out);
// Window means and inverse norms of the FP32 forms, with `pad` zeros behind the
// series and both; nchg (n ints) and tot (n / 256 + 2 ints) are used by windows too
// long for one block's shared memory.  Returns the number of launches.
int launch_fp32_stats(double* A, int64_t m, int64_t PL, int64_t pad, int* nchg, int* tot, double* mean,
                      double* norm, cudaStream_t s);
void configure_stats();  // per-device setup, before a stream capture

// ---- FP64 diagonal-band join (mp_join_fp64.cu) ------------------------------
// Diagonal g (g_lo <= g < g_hi) meets column j in row r = j + g, for
// j < Tbase - g.  The reference's block geometry (blocks of B diagonals
// starting at blk_origin, triangle length T = Tbase - block start) decides
// per cell whether the fused or the separately rounded arithmetic applies.
//
// Bands cut into tiles of L columns (fp64_split_plan says when).  A tile starts
// from its diagonals' running dot products at its first column, which
// launch_fp64_seeds computes beforehand.  A row that several tiles of a band meet
// keeps the whole band's choice: the tiles leave their best cells of it in
// seam_s / seam_j, and fp64_seam_kernel merges the best of them.
struct Fp64Split {
    int64_t L;             // columns per tile, a multiple of kFp64SplitUnit; 0: whole bands
    int64_t nseg;          // tiles of the longest band
    int64_t seg_per_pair;  // tile numbering: see tile_of_pair
    int64_t ntiles;
    double* seeds;         // [nseg - 1][g_hi - g_lo]: dot product at column (s + 1) L
    double* seam_s;        // [ntiles][fp64_seam_rows] best score of a seam row of the tile ...
    int* seam_j;           // ... and its column, -1: none
};
constexpr int64_t kFp64SplitUnit = 16;
// Rows of a tile that a tile of its band before or after it may meet, too: the first and
// the last `span` (= 32R) of its L + span.  Their number, and row t's place among them.
__host__ __device__ inline int64_t fp64_seam_rows(int64_t L, int64_t span) { return span + (L < span ? L : span); }
__host__ __device__ inline int64_t fp64_seam_slot(int64_t t, int64_t L, int64_t span) {
    return t < span || L < span ? t : t - L + span;
}
// Number of a tile in a list of band pairs (k, nbands - 1 - k), whose lengths are
// nearly complementary: pair p = lt / seg_per_pair holds the tiles of K columns of
// band p, then those of band nbands - 1 - p.  False for the unused tail of a pair.
// (Host-callable too, so the tile space can be checked without a GPU.)
__host__ __device__ inline bool tile_of_pair(int64_t lt, int64_t PL, int64_t g_lo, int64_t K,
                                             int64_t nbands, int64_t seg_per_pair, int64_t span,
                                             int64_t& band, int64_t& seg) {
    const int64_t p = lt / seg_per_pair;
    int64_t s = lt % seg_per_pair;
    const int64_t nseg0 = (PL - (g_lo + p * span) + K - 1) / K;
    if (s < nseg0) {
        band = p;
        seg = s;
        return true;
    }
    s -= nseg0;
    const int64_t p2 = nbands - 1 - p;
    if (p2 <= p) return false;
    const int64_t nseg1 = (PL - (g_lo + p2 * span) + K - 1) / K;
    band = p2;
    seg = s;
    return s < nseg1;
}
// The gate's tests are integer ones, on high words: those of non-negative doubles order
// like the doubles.  (Host-callable, so the rule can be checked without a GPU.)
__host__ __device__ inline int high_word(double x) {
#ifdef __CUDA_ARCH__
    return __double2hiint(x);
#else
    int64_t b;
    std::memcpy(&b, &x, 8);
    return (int)(b >> 32);
#endif
}
__host__ __device__ inline double from_words(int hi, int lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(hi, lo);
#else
    const int64_t b = (int64_t)(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo);
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// A window's scale s = 1 / deviation and mean term w for which s, its products and
// quotients with w stay far from the ends of a double's range (a small w may vanish:
// what it adds lies below the gates' slack).
__host__ __device__ inline bool fp64_ordinary(double s, double w) {
    return (unsigned)(high_word(s) - ((1023 - 450) << 20)) < (unsigned)(900 << 20) &&
           (high_word(w) & 0x7fffffff) < ((1023 + 200) << 20);
}
// A constant window with a mean: s = +inf, w = +-inf.
__host__ __device__ inline bool fp64_flat(double s, double w) {
    return s > DBL_MAX && (w > DBL_MAX || w < -DBL_MAX);
}
// A window without a finite score: its scores are NaN, or with a constant window NaN or
// infinite.  No score of it is between a finite bound and the largest double, so that
// serves as the bound of every one of its cells, and its gate stays shut for finite ones.
__host__ __device__ inline bool fp64_degenerate(double s, double w) {
    return s != s || w != w || fp64_flat(s, w);
}
__host__ __device__ inline double fp64_bound(double threshold, double s, double w) {
    return !fp64_ordinary(s, w) && fp64_degenerate(s, w) ? DBL_MAX : threshold;
}
// A column's mean term in the FP64 join's gate, which tests s' (q s - w W') in place of
// the score q (s s') - w w': W' = w' / s'.  A constant column's scores are -inf, NaN, or
// +inf where w w' < 0; with the largest double as W' the gate's value is positive there.
__host__ __device__ inline double fp64_gate_mean(double s, double w) {
    if (fp64_ordinary(s, w)) {
        const double x = w / s;
        return x != 0.0 || w == 0.0 ? x : copysign(DBL_MIN, w);  // its product with an infinite term keeps its sign
    }
    if (fp64_flat(s, w)) return w > 0.0 ? DBL_MAX : -DBL_MAX;
    return w != w ? w : 0.0;  // the gate stands open (fp64_gate_error), or the score is NaN
}
// A bound's gate: minus the high word of a value below it by more than the rounding
// of the gate's values (kFp64GateSlack m, and 2^-34 of the bound).  A negative bound lets
// every cell through; past kFp64GateEnd, where a product may leave the range of doubles
// (and the gate's value counts as the largest one), a bound's gate is that end's.
constexpr double kFp64GateSlack = 0x1p-25;
constexpr int kFp64GateEnd = (1023 + 500) << 20;
__host__ __device__ inline int fp64_gate(double bound, double m) {
    const int h = high_word(fma(bound, 1.0 - 0x1p-34, -kFp64GateSlack * m));
    return h > 0 ? -(h < kFp64GateEnd ? h : kFp64GateEnd) : 0;
}
// The same from the bound's high word h alone, a unit lower: from m / 16 on a unit is
// more than the slack.
__host__ __device__ inline int fp64_gate_high_from(double m) { return high_word(m * 0x1p-4) + 1; }
__host__ __device__ inline int fp64_gate_high(int h, int from) {
    return h >= from ? 1 - (h < kFp64GateEnd ? h : kFp64GateEnd) : 0;
}
// Added to a score's high word, kFp64NoNan takes a NaN (0x7ff8 or above, or its negative)
// to a negative number or 0 and leaves the order of all other values.  A score passes a
// gate if fp64_cell_high + fp64_cell_gate >= kFp64Pass (the largest sum is 0x7fffffff).
constexpr int kFp64NoNan = 0x80000, kFp64Pass = kFp64NoNan - 1;
__host__ __device__ inline int fp64_cell_high(int h) {
#ifdef __CUDA_ARCH__
    return __viaddmax_s32(h, kFp64NoNan, 0);
#else
    const int x = (int)((unsigned)h + (unsigned)kFp64NoNan);
    return x > 0 ? x : 0;
#endif
}
__host__ __device__ inline int fp64_cell_gate(int gate) { return gate < 0 ? gate - 1 : kFp64Pass; }
// The same from the high word of a best score of the same arithmetic, which needs no slack.
__host__ __device__ inline int fp64_best_gate(int h) { return h > 0 ? -h - 1 : kFp64Pass; }
// High word of the gate's value, from the largest high word among a column's
// q s - w W' (0 if all are negative): rounded up, an infinity or NaN as the largest
// double.  The cell passes if the sum with its bound's gate is not negative.
__host__ __device__ inline int fp64_gate_value(int top, double s) {
    return high_word(from_words(top < 0x7fefffff ? top : 0x7fefffff, -1) * s);
}
// What the gate's value may lie below a cell's score because of a window with scale s
// and mean term w, as the high word of an upper bound; an infinite one lets every cell
// through.  With u = 2^-53, the score is off its exact value S by 2u|S| + 2u|w w'|,
// the gate's value by 3u|S| + 2u|w w'|; |w w'| <= (w^2 + w'^2) / 2 parts the rounding
// of the mean terms between the two windows, 2^-51 w^2 for each with room.
__host__ __device__ inline int fp64_gate_error(double s, double w) {
    if (fp64_ordinary(s, w)) {
        const int h = high_word(w * w) + 1 - (51 << 20);
        return h > 0 ? h : 0;
    }
    // NaN never selects; infinite terms give the score's own infinities and NaN
    return fp64_degenerate(s, w) ? 0 : 0x7ff00000;
}
// Errors up to here are within the gates' slack.
__host__ __device__ inline int fp64_gate_errfree(double m) { return high_word(kFp64GateSlack / 8 * m); }
// For larger ones (err: the larger of a pass's rows' and columns'): whether the largest
// value over its gate lets the pass open when every gate lies lower by the units that
// take the smallest bound (gate g) below it by both errors; the units of larger bounds
// are at least as wide.
__host__ __device__ inline bool fp64_gate_lowered(int g, int err, int over) {
    if (err >= 0x7ff00000) return true;
    const int h = high_word(from_words(-g, 0) - 2.0 * from_words(err, 0));
    return h <= 0 || over >= h + g - 1;
}
struct Fp64BandParams {
    const double4* colrec;  // colrec[j] = {A_hor[j], A_hor[j+m], s_hor[j], mu_hor[j]}
    const double4* rowrec;  // rowrec[r] = {A_vert[r], A_vert[r+m], s_vert[r], mu_vert[r]}
    const double* colgate;  // colgate[j] = fp64_gate_mean(s_hor[j], mu_hor[j]), Tbase values
    const double* qt0;      // qt0[g - g_lo]: running dot product at j = 0
    double* qt_out;         // optional: dot product after the last cell, per diagonal
    int64_t g_lo, g_hi, nbands;
    int64_t blk_origin, B, Tbase;
    unsigned long long* kexact;  // [shards][key_stride] ordered score, max-merged
    unsigned long long* kidx;    // [shards][key_stride] truncated score | neighbour
    int64_t key_stride;
    int shards;
    int64_t row_key_off, col_key_off;  // key slot of row r / column j
    int64_t row_nb_off, col_nb_off;    // neighbour written for column j / row r
    double m;
    double floor;  // only scores strictly above it are merged (-1: reference init)
    int idx_bits;
    long long key_vlo;  // bit pattern of the index key's lower range end (idx_key_f64)
    // Selection thresholds, one per key slot plus kFp64ThrPad slots of padding
    // (initialised to -DBL_MAX).  Every merge raises thr[slot] to a value a
    // little below the merged score (fp64_threshold_below); a cell whose score
    // does not exceed its row's and its column's thresholds can change neither
    // key, so a column step whose cells all fall below them skips selection.
    double* thr;
    double thr_eps;   // relative margin, wider than the index key's resolution
    double thr_tiny;  // absolute margin near v = m - score = 0
    unsigned* counter;  // work handed out beyond the first wave (zeroed by the launch)
    int64_t spread;     // set by the launch: every spread-th band is in the first wave
    Fp64Split split;    // split.L > 0: bands cut into tiles of L columns
};
// Order of the bands: every spread-th band first (longest to shortest), then
// the others, longest first.
__host__ __device__ inline int64_t fp64_band_of(int64_t rank, int64_t nbands, int64_t spread) {
    const int64_t first = (nbands + spread - 1) / spread;
    if (rank < first) return rank * spread;
    rank -= first;
    return rank / (spread - 1) * spread + 1 + rank % (spread - 1);
}
constexpr int kFp64WarpsPerBlock = 4;
constexpr int64_t kFp64ThrPad = 64 * 8 + 64;  // >= the 34R + R rows staged past a band's end
// Threshold stored after merging `score` (see Fp64BandParams::thr): below the
// score by more than the index key's resolution, so every cell whose index key
// could still tie or beat the key of a merged cell exceeds it.  Host-callable
// so the margin can be checked without a GPU.
__host__ __device__ inline double fp64_threshold_below(double score, double m, double eps,
                                                       double tiny) {
    const double v = m - score > 0.0 ? m - score : 0.0;
    return m - (v * (1.0 + eps) + tiny);
}
// Margins for a key with idx_bits index bits: the index key keeps 57 - idx_bits
// mantissa bits of v, i.e. a relative resolution of 2^(idx_bits - 57); eps is
// eight times that, tiny covers |v| near 0, where the key clamps.
inline double fp64_threshold_eps(int idx_bits) { return std::ldexp(1.0, idx_bits - 54); }
inline double fp64_threshold_tiny(double m) { return std::ldexp(m, -40); }
template <int R>
void launch_fp64_band(const Fp64BandParams& P, cudaStream_t s);
// Split plan of a band join over diagonals [g_lo, g_hi) of Tbase columns (L = 0:
// whole bands), with tiles long enough for buffers of `room` bytes; the bytes its buffers
// need, and the buffers carved from `base`.
Fp64Split fp64_split_plan(int64_t Tbase, int64_t g_lo, int64_t g_hi, int R, size_t room = SIZE_MAX);
size_t fp64_split_bytes(const Fp64Split& S, int64_t ndiag, int R);
void fp64_split_carve(Fp64Split& S, int64_t ndiag, int R, char* base);
// Running dot products at the tiles' first columns: Ah the series along columns,
// Av along rows (nh and nv values; zero is read past them), P.qt0 the dot products
// at column 0.
// X.n > 0: one more block takes the reference-order prefix sums of X.A.
struct PrefixSums {
    const double* A;
    int64_t n;
    double *cs, *cs2;
};
void launch_fp64_seeds(const Fp64BandParams& P, const double* Ah, int64_t nh, const double* Av,
                       int64_t nv, int64_t m, const PrefixSums& X, cudaStream_t s);

// ---- FP32 re-anchored tile join (mp_join_fp32.cu) ---------------------------
// One series of a (batched) join.  Its tiles are numbered
// [tile_begin, tile_begin + npairs * seg_per_pair) in the launch's tile space;
// a launch that runs only a slice of them (the request server's epochs) starts
// at the series' local tile tile_skip.
struct Fp32TileParams {
    const float4* rowrec;  // pairs (x[j], x[j+H]) of df, dg, nn; 2 float4 per row
    const float4* colrec;  // duplicated, negated column terms; 2 float4 per column
    const double* A;       // series (FP64) for the anchors
    const double* mean;    // window means (FP64)
    int64_t m, PL;
    int64_t g_lo, g_hi;    // diagonals evaluated
    int64_t K;             // columns per tile = re-anchor interval
    int64_t nbands;        // bands of 32R diagonals
    int64_t seg_per_pair;  // tiles per band pair (k, nbands-1-k), max over pairs
    int64_t tile_begin;    // first tile of this series in the launch
    int64_t tile_skip;     // local tile that launch tile tile_begin stands for (0: all)
    unsigned long long* key;  // [PL] (ordered u << 32 | neighbour or group), min-merged
    // Guarded form only (all null otherwise): hazard[w] = number of hazard
    // windows among [0, w) (PL + 1 entries); FP64 inverse norms and
    // recurrence terms for the FP64 tiles.
    const int* hazard;
    const double* norm;
    const double* df;
    const double* dg;
};
#ifdef __CUDACC__
// A row or column record in global memory: (x[j], x[j+4]) pairs of df, dg, nn for
// rows, (-df, -df, -dg, -dg, nn, nn, 1/nn, 1/nn) for columns.  Record i from `base` on:
// with 2^28 columns between re-anchors its offset passes 32 bits.
constexpr int kFp32RecFloats = 8;
__host__ __device__ __forceinline__ const float* fp32_record(const float* base, int64_t i) {
    return base + i * kFp32RecFloats;
}
// Local tile lt of a series -> (band, column segment), see tile_of_pair.
__host__ __device__ __forceinline__ bool fp32_tile_of(const Fp32TileParams& P, int64_t lt, int64_t span,
                                             int64_t& band, int64_t& seg) {
    return tile_of_pair(lt, P.PL, P.g_lo, P.K, P.nbands, P.seg_per_pair, span, band, seg);
}
// Guarded form: does the tile (band start gb, columns [j0, j1)) touch a
// hazard window, as a column or as a row (rows j + g, g in [gb, gb + span))?
__device__ __forceinline__ bool fp32_tile_hazardous(const Fp32TileParams& P, int64_t gb, int64_t j0,
                                                    int64_t j1, int span) {
    const int64_t rs = min(j0 + gb, P.PL), re = min(j1 + gb + span, P.PL);
    return (P.hazard[j1] - P.hazard[j0]) > 0 || (P.hazard[re] - P.hazard[rs]) > 0;
}

// Records (count of them), keys (set to init), and optionally the launch's only
// descriptor P -> *desc and its tile counter.
__global__ void pack_fp32_kernel(const double* A, int64_t m, int64_t PL, int H, int64_t count,
                                 const double* mean, const double* norm, float4* rowrec, float4* colrec,
                                 unsigned long long* key, unsigned long long init, const Fp32TileParams P,
                                 Fp32TileParams* desc, unsigned long long* counter);

// A window's key before any candidate: no neighbour, at u = 1 + 1/m (`init`).  A flat
// window (NaN inverse norm), which never gets one, starts at the largest key, so that the
// gates need not wait for its first.
constexpr unsigned long long kFp32FlatKey = ~0ull;
__host__ __device__ __forceinline__ unsigned long long fp32_first_key(unsigned long long init, double norm) {
    return norm == norm ? init : kFp32FlatKey;
}
// Bit pattern of the largest distance u that still concerns a key's window, from the
// key's high word: 0 where the key's own is negative (any such cell goes on), and for a
// flat window.  With `tags`, just above every tagged distance that could tie the key
// (2^-15 steps).
__host__ __device__ __forceinline__ unsigned fp32_key_bound(unsigned hi, bool tags) {
    if (!(hi & 0x80000000u)) return 0u;
    if (tags) return ((hi & 0x7fffff00u) + 0x100u) & 0x7fffffffu;  // a flat window's wraps to 0
    return hi == 0xffffffffu ? 0u : hi & 0x7fffffffu;
}

// FP32 profile keys, min-merged: (ordered u << 32) | neighbour.  With group
// keys (the guarded form) the tile kernel finds a minimum's lane but not which
// of the lane's R diagonals holds it, so its keys name a group of adjacent
// candidate neighbours instead: bit 31 of the low word set, the group's first
// candidate in bits 0..30, and (count - 1) in the low 3 bits of the high word
// -- below the form's 2^-15 resolution of u, which keeps 0x80 in the low byte
// of u's pattern.  Keys with bit 31 clear (FP64 tiles, exact pairs, the
// initial key) name the neighbour itself.
constexpr unsigned kFp32GroupBit = 0x80000000u;
// A group key is resolved among its candidates and kPickSpan more on each
// side (FP32 ranking noise between adjacent diagonals does not stop at a
// group's edge): of the candidates q in [lo, lo + n) (n <= kPickSlots) that
// are partners of window i in the join (0 <= q < PL, g_lo <= |i - q| < g_hi),
// the one whose window has the largest centred FP64 correlation with window
// i, ties to the smaller index; NaN (flat) candidates never win; -1 when none
// qualifies.  A, mean and norm (inverse centred norms) as in the tile kernel;
// A holds at least kPickSlots - 1 values of padding past the series.  About
// kPickSlots * m FMAs.  Host-callable too, so the candidate rules can be
// checked without a GPU.
constexpr int kPickSpan = 4;
constexpr int kPickSlots = 8 + 2 * kPickSpan;
__host__ __device__ inline double pick_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
__host__ __device__ inline int64_t fp32_pick_neighbour(const double* A, const double* mean,
                                                       const double* norm, int64_t m, int64_t PL,
                                                       int64_t g_lo, int64_t g_hi, int64_t i,
                                                       int64_t lo, int n) {
    constexpr int W = kPickSlots;
    const int64_t hi = lo + (int64_t)n < PL ? lo + (int64_t)n : PL;
    lo = lo > 0 ? lo : 0;
    double c[W], w[W];
#pragma unroll
    for (int a = 0; a < W; ++a) c[a] = 0.0;
    const double mi = mean[i];
    double sx = 0.0;
#pragma unroll
    for (int a = 0; a < W - 1; ++a) w[a] = A[lo + a];
    int64_t t = 0;
    for (; t + W <= m; t += W) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            w[(k + W - 1) % W] = A[lo + t + k + W - 1];
            const double x = A[i + t + k] - mi;
            sx += x;
#pragma unroll
            for (int a = 0; a < W; ++a) c[a] = pick_fma(x, w[(k + a) % W], c[a]);
        }
    }
    for (; t < m; ++t) {
        const double x = A[i + t] - mi;
        sx += x;
#pragma unroll
        for (int a = 0; a < W; ++a) c[a] = pick_fma(x, A[lo + t + a], c[a]);
    }
    // sum_t x_t (A[q+t] - mean_q) = c - mean_q * sum_t x_t; the common factor
    // norm[i] > 0 does not change the ranking
    int64_t best = -1;
    double bs = -__builtin_huge_val();
#pragma unroll
    for (int a = 0; a < W; ++a) {
        const int64_t q = lo + a;
        const int64_t g = q > i ? q - i : i - q;
        if (q < hi && g >= g_lo && g < g_hi) {
            const double sc = (c[a] - mean[q] * sx) * norm[q];
            if (sc > bs) {
                bs = sc;
                best = q;
            }
        }
    }
    return best;
}
#endif
// Persistent launch over `nseries` descriptors (device array) holding `total`
// tiles; warps take tiles from *counter (zeroed by the caller beforehand).
// group: the keys name candidate groups (see kFp32GroupBit) instead of
// neighbours, which the finalisation resolves in FP64 (not with kFp32Mixed).
enum Fp32Way { kFp32Dense, kFp32Gate, kFp32Mixed };
template <int R>
void launch_fp32_join(const Fp32TileParams* series_dev, int nseries, int64_t total,
                      unsigned long long* counter, cudaStream_t s, Fp32Way way, bool group = false);
// Whether a join's passes go behind the gate (mp_join_fp32.cu) or all select.  A
// row's minimum falls about as often as a record in a random sequence, log of the
// candidates, each time over a run of lags that grows shorter with the window; the
// gate opens for the loosest of 24 rows and 16 columns, which lie further apart
// with short windows.  Random walks, K = 1024, gate / every pass selecting (ms):
//   m = 64    n = 500,000 41.9 / 39.0
//   m = 96    262,144 10.2 / 10.8     500,000 35.4 / 39.1
//   m = 128   65,536 0.76 / 0.73      131,072 2.48 / 2.76     500,000 32.1 / 39.3
//   m = 160   32,768 0.25 / 0.26      65,536 0.71 / 0.73      262,144 8.7 / 10.9
//   m = 256   16,384 0.12 / 0.10      32,768 0.24 / 0.30      131,072 2.19 / 2.80
//   m = 1024  16,384 0.13 / 0.11      32,768 0.25 / 0.29
// (30,000 / 170: 0.24 / 0.18.)  Up to about 30,700 samples the selecting passes' tiles are one
// wave of their 1,776 resident warps; the gate, which spreads over more, gains nothing there.
// Other data moves the lines: noisy steps of 150 samples, m = 96 to 130 0.86 to 0.89 times as
// fast behind the gate, white noise 1.2 to 1.3 times.
__host__ __device__ inline bool fp32_gate_pays(int64_t m, int64_t PL) {
    return m >= 96 && PL >= (m >= 160 ? 30700 : m >= 128 ? 90000 : 200000);
}
// The way of a launch over these series.
inline Fp32Way fp32_way_of(const Fp32TileParams* P, size_t n) {
    size_t gate = 0;
    for (size_t i = 0; i < n; ++i) gate += fp32_gate_pays(P[i].m, P[i].PL);
    return gate == 0 ? kFp32Dense : gate == n ? kFp32Gate : kFp32Mixed;
}
template <int R>
void configure_fp32_join();
// Guarded form (mp_guard.cu): hazard windows and the FP64 pass over their tiles.
#ifdef __CUDACC__
// The hazard rule, host-callable so that it can be checked without a GPU.
// Window w is a hazard when it is flat (NaN inverse norm) or its inverse norm
// exceeds kGuardRatio times the smallest inverse norm among windows
// [w - (blk - 1), w]; that minimum comes from a van Herk / Gil-Werman sliding
// minimum: prefix and suffix minima within blocks of blk windows (fmin ignores
// NaN, so flat windows never lower it).
constexpr double kGuardRatio = 16.0;
// Block b: pre[i] = min nn[b*blk .. i], suf[i] = min nn[i .. end of block b].
__host__ __device__ inline void hazard_block_minima(const double* nn, int64_t PL, int64_t blk,
                                                    int64_t b, double* pre, double* suf) {
    const int64_t i0 = b * blk;
    if (i0 >= PL) return;
    const int64_t i1 = i0 + blk < PL ? i0 + blk : PL;
    double v = nn[i0];
    for (int64_t i = i0; i < i1; ++i) {
        v = fmin(v, nn[i]);
        pre[i] = v;
    }
    v = nn[i1 - 1];
    for (int64_t i = i1 - 1; i >= i0; --i) {
        v = fmin(v, nn[i]);
        suf[i] = v;
    }
}
// 1 when window w (< PL) is a hazard, from the block minima above.
__host__ __device__ inline int hazard_flag(const double* nn, const double* pre, const double* suf,
                                           int64_t blk, int64_t w) {
    const int64_t look = blk - 1;
    double mn;
    if (w < look) {
        mn = pre[w];
    } else {
        const int64_t a = w - look;
        mn = (a % blk == 0) ? pre[w] : fmin(suf[a], pre[w]);
    }
    const double x = nn[w];
    return (x != x || x > kGuardRatio * mn) ? 1 : 0;
}
#endif
__global__ void hazard_block_minima_kernel(const double* nn, int64_t PL, int64_t blk, double* pre,
                                           double* suf);
__global__ void hazard_flags_kernel(const double* nn, const double* pre, const double* suf,
                                    int64_t PL, int64_t blk, int* flag);
__global__ void guard_terms_kernel(const double* A, int64_t m, int64_t PL, const double* mean,
                                   double* df, double* dg);
// Persistent FP64 pass over the same tile space as launch_fp32_join; only
// tiles that touch a hazard window do work (counter zeroed beforehand).
template <int R>
void launch_fp64_guard(const Fp32TileParams* series_dev, int nseries, int64_t total,
                       unsigned long long* counter, cudaStream_t s);
// Near-duplicate pass of the guarded form (mp_guard.cu).
struct NearDupParams {
    const double* A;
    const double* mean;
    const double* norm;  // FP64 inverse norms (NaN: flat)
    int64_t m, PL;
    int64_t g_lo, g_hi;  // pairs on diagonals [g_lo, g_hi) only
    const int* list;     // the collected windows
    int64_t count;
    unsigned long long* key;
    float ulim;
};
__global__ void neardup_collect_kernel(const unsigned long long* key, int64_t PL, float tau,
                                       unsigned long long init, int* list, int* count, int cap);
__global__ void neardup_reset_kernel(const int* list, int count, unsigned long long* key,
                                     unsigned long long init);
__global__ void neardup_pairs_kernel(const NearDupParams P);
// Re-anchor interval K (columns per FP32 tile) from the caller's value: 1024
// when not positive, at most 2^31 (every profile is shorter, so a longer
// interval changes nothing and the rounding below cannot overflow), rounded
// up to a multiple of the R columns a chunk processes.
inline int64_t reanchor_interval(int64_t k, int R) {
    int64_t K = k > 0 ? k : 1024;
    if (K > (int64_t(1) << 31)) K = int64_t(1) << 31;
    return ((K + R - 1) / R) * R;
}
// Tile count and seg_per_pair of one series (host helper).
void fp32_tile_plan(int64_t PL, int64_t g_lo, int64_t g_hi, int64_t K, int R, int64_t& nbands,
                    int64_t& seg_per_pair, int64_t& ntiles);

// ---- PreSCRIMP (mp_prescrimp.cu) -------------------------------------------------
struct PreScrimpParams {
    const double* A;      // series, n samples
    const double* mean;   // window means (reference order)
    const double* sigma;  // window standard deviations (reference order)
    int64_t n, m, PL, excl;
    int64_t step;         // floor(stride * m): query i_t = t * step
    int64_t Q;            // number of queries
    unsigned long long* kex;  // [PL] ordered distance, min-merged
    unsigned long long* kix;  // [PL] ordered distance (high bits) | neighbour, min-merged
    unsigned long long* rex;  // [Q] a query's own best (distance)
    unsigned long long* rix;  // [Q] ... (neighbour)
    int idx_bits;
};
// Whether the windows i and j lie within the exclusion zone (ScrimpppOrig.cpp:190-193).
// (Host-callable, so the rule can be checked without a GPU.)
__host__ __device__ inline bool prescrimp_excluded(unsigned i, unsigned j, unsigned excl) {
    return (j > i ? j - i : i - j) < excl;
}
__global__ void orig_stats_kernel(const double* cs, const double* cs2, int64_t PL, int64_t m,
                                  double* mean, double* sigma);
__global__ void prescrimp_keys_init_kernel(unsigned long long* a, int64_t count);
__global__ void prescrimp_finalize_kernel(const unsigned long long* kex,
                                          const unsigned long long* kix, int64_t PL, int idx_bits,
                                          double* d2, int64_t* idx);
// Query rows then diagonal walks (2 launches).
void launch_prescrimp(const PreScrimpParams& P, cudaStream_t s);

// ---- finalisation (mp_finalize.cu) -------------------------------------------
__global__ void init_keys_kernel(unsigned long long* k, int64_t count, unsigned long long v);
__global__ void finalize_fp64_kernel(const unsigned long long* kexact, const unsigned long long* kidx,
                                     int64_t key_stride, int shards, int64_t PL, double m,
                                     int idx_bits, double* d2, int64_t* idx);
__global__ void finalize_fp32_kernel(const unsigned long long* key, int64_t PL, double m,
                                     const double* A, const double* mean, const double* norm,
                                     int refine, double* d2, int64_t* idx);
__global__ void finalize_fp32_guarded_kernel(const unsigned long long* key, int64_t PL, double m,
                                             const double* A, const double* mean, const double* norm,
                                             int64_t g_lo, int64_t g_hi, double* d2, int64_t* idx);
__global__ void block_keys_init_kernel(const double* prof, int64_t count, unsigned long long* kexact,
                                       unsigned long long* kidx);
__global__ void block_finalize_kernel(const unsigned long long* kexact, const unsigned long long* kidx,
                                      int64_t key_stride, int shards, int64_t count, int idx_bits,
                                      double* prof, int64_t* idx);

}  // namespace mpgpu
