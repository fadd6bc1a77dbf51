// FP32 re-anchored tile join.
//
// The distance matrix is cut into tiles of 32*R adjacent diagonals (one
// band) by K columns.  A warp owns one tile: lane l owns diagonals
// g0 + a (a < R, g0 = band start + l*R), all lanes walk the tile's columns
// together.
//
//  anchor     at the tile's first column j0 each lane computes the exact
//             covariance of its R window pairs in FP64:
//               cov = sum_k A[j0+k]*A[j0+g+k] - m*mean[j0]*mean[j0+g]
//             (the re-anchor; one per K recurrence steps);
//  recurrence the centred update of SCAMP (Zimmerman et al., SoCC 2019),
//               cov(j+1, r+1) = cov(j, r) + df[j]*dg[r] + df[r]*dg[j],
//             in FP32 with fused multiply-adds;
//  distance   u = 1 - cov*nn[j]*nn[r] (= d^2 / 2m) as a single fused op;
//  min/argmin the low 8 bits of u's bit pattern are replaced by the cell's
//             position in the band (lane<<3 | a), so one float min tracks
//             value and origin at once (2^-15 relative resolution, far
//             inside the 1e-4 target).  A row's best tagged distance sits in
//             the warp's shared memory until the warp's lowest lane has met
//             the row; a column's warp minimum is one REDUX instruction.
//             Finished rows/columns are merged into the profile with a 64-bit
//             atomicMin on (ordered u, neighbour).
//  gate       almost no cell can lower either minimum, so a pass of 16 columns
//             first runs the recurrence with one more fused operation per cell,
//             whose sign says whether the distance is at or below the loosest
//             bound that the lane meets in the pass: its rows' best distances,
//             which start just above the rows' keys as they stand in global
//             memory (a stale key is only a looser start), and the columns'
//             keys.  A cell that passes neither can change neither key.  When
//             some lane has a cell that may, the pass is evaluated again with
//             the selection (dense_pass); a pass that lowered something is
//             followed by one with the selection straight away, so data that
//             selects everywhere costs little more than the selection itself.
//  group keys (the guarded form) a lane takes plain float minima over its
//             own cells, and only the lane's results carry the lane number
//             in their low 8 bits (one tag per row or column, not per cell);
//             a key then names the winning lane's R adjacent candidate
//             neighbours, among which the finalisation picks with FP64 dot
//             products (fp32_pick_neighbour) -- which also removes FP32
//             ranking noise between adjacent diagonals.
//
// What bounds it: instruction issue and register reads.  Behind the gate a column of
// a lane's 8 cells takes 24 fused multiply-adds, 5 others for the test and 3
// shared-memory reads (12 bytes a lane), 53 cycles of a scheduler; a fused operation
// with three different operands takes the register file 1.5 cycles (measured;
// packed f32x2 pairs cost the same words, their pair records twice the
// shared-memory bandwidth, and minima in place of sign bits three cycles each).
// n = 1,048,576, m = 256, K = 1024: 127 ms (100 the columns, 10 the passes' ends, 8
// passes evaluated again, the rest anchors), 178 ms with every pass selecting,
// which stays the better way for short windows and short series (fp32_gate_pays).
// Both kinds of pass are loops over two halves of 8 columns: unrolled over 16 they
// wait for instructions where passes of both kinds follow each other (n = 65,536, m =
// 400: 0.74 -> 0.64 ms, 262,144 / 256: 8.9 -> 8.3 ms).
//
// Reference semantics kept: strict improvement over the initial score -1
// (u < 1 + 1/m), NaN never wins (a zero-variance window has nn = NaN).
#include <algorithm>
#include <atomic>

#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_tile.cuh"

namespace mpgpu {

namespace {

constexpr int kRecFloats = kFp32RecFloats;
constexpr int kR = kTileR;  // 8: tags of 3 + 5 bits

constexpr unsigned kTagMask = 0xffu;
constexpr float kInf = __builtin_huge_valf();

// Floats between the ring's groups of 8 rows (48 bytes), so that the 8 lanes of a
// quarter-warp taking a group each with 16-byte accesses hit 8 distinct groups of
// 4 banks (a 32-byte stride would pair them up).
constexpr int kRowStride = 12;

// 4-byte copy global -> shared that completes asynchronously.
__device__ __forceinline__ void cp_async4(float* dst_smem, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ float tag_key(float u, unsigned tag) {
    return __uint_as_float((__float_as_uint(u) & ~kTagMask) | tag);
}
__device__ __forceinline__ float untag_value(unsigned bits) {
    return __uint_as_float((bits & ~kTagMask) | 0x80u);
}
// u with the lane number in its low 8 bits (group keys: a lane's minima only).
__device__ __forceinline__ float tag_lane(float u, unsigned lane) {
    return __uint_as_float((__float_as_uint(u) & ~kTagMask) | lane);
}

template <bool GROUP>
__device__ __forceinline__ float lane_min(float v, int lane) {
    return GROUP ? tag_lane(v, (unsigned)lane) : v;
}

// Group keys: merges (u, candidates [base, base + count)) unless u is not
// below the initial score's ulim.
__device__ __forceinline__ void merge_group(unsigned long long* key, float u, int64_t base,
                                            int count, unsigned ulim_ord) {
    const unsigned hi = (ord_f32(u) & ~kTagMask) | 0x80u | (unsigned)(count - 1);
    if (hi < ulim_ord)
        atomicMin(key, ((unsigned long long)hi << 32) | kFp32GroupBit | (unsigned long long)base);
}
// Row r's minimum over the band, tagged with its lane L: the cells of lane L
// in row r are (j = r - g, g = gL + a) for a < kR with g < g_hi and j >= 0,
// gL = gb + L*kR, i.e. the columns [r - gL - amax, r - gL].
__device__ __forceinline__ void flush_row_group(const Fp32TileParams& P, float v, int64_t r,
                                                int64_t gb, unsigned ulim_ord) {
    const unsigned bits = __float_as_uint(v);
    const float u = untag_value(bits);
    if (!(u < kInf)) return;  // no cell (kInf or a NaN pattern)
    const int64_t gL = gb + (int64_t)(bits & kTagMask) * kR;
    const int64_t amax = min(min((int64_t)kR - 1, P.g_hi - 1 - gL), r - gL);
    merge_group(P.key + r, u, r - gL - amax, (int)amax + 1, ulim_ord);
}
// Column j's minimum over the band, tagged with its lane L: the candidates
// are rows j + gL + a, a < kR, on diagonals < g_hi and rows < PL.
__device__ __forceinline__ void flush_col_group(const Fp32TileParams& P, unsigned bits, int64_t j,
                                                int64_t gb, unsigned ulim_ord) {
    const float u = untag_value(bits);
    if (!(u < kInf)) return;
    const int64_t gL = gb + (int64_t)(bits & kTagMask) * kR;
    const int64_t cnt = min(min((int64_t)kR, P.g_hi - gL), P.PL - j - gL);
    merge_group(P.key + j, u, j + gL, (int)cnt, ulim_ord);
}

__device__ __forceinline__ void flush_row(const Fp32TileParams& P, float v, int64_t r,
                                          int64_t gb, float ulim) {
    const unsigned bits = __float_as_uint(v);
    const float u = untag_value(bits);
    if (u < ulim) {
        const unsigned t = bits & kTagMask;
        const int64_t j = r - (gb + t);  // lane << 3 | a is the diagonal's place in the band
        atomicMin(P.key + r, ((unsigned long long)ord_f32(u) << 32) | (unsigned long long)j);
    }
}

static_assert(kAnchorBytes <= kRecRingBytes, "anchor staging fits the record ring");

// ---- every pass with the selection (see fp32_gate_pays) ----------------------
// A row record in memory: 32 bytes.
struct RowRec {
    float4 dfdg;  // (df[j], df[j+4], dg[j], dg[j+4])
    float4 nn1;   // (nn[j], nn[j+4], 1, 1)
};
// The part of a row record a lane keeps in registers (the constant pair stays
// behind: one shared (1, 1) operand serves every fused distance).
struct DenseWin {
    float4 dfdg;
    float2 nn;
};
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }
static_assert(sizeof(RowRec) == 4 * kRecFloats, "row record is 32 bytes");

// Row-partial ring: 34 chunks of 8 rows, 12 floats apart (48 bytes), so that
// the 8 lanes of a quarter-warp merging their chunks with 16-byte accesses
// hit 8 distinct groups of 4 banks (a 32-byte stride would pair them up).
constexpr int kRowChunks = 34;

// 16-byte copy global -> shared that completes asynchronously (cp.async.cg:
// cached in L2 only); both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(char* dst_smem, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// One chunk = R consecutive columns.  Per column: R cells per lane, the
// lane's column minimum, then one warp-wide REDUX; lane OFF + b keeps the
// result of column b so the column flushes happen once per chunk pair, with
// no divergent branch between steps (consecutive steps can overlap).  Row
// partials live in a 2R-entry circular register array; OFF (0 or R) is the
// chunk's rotation, so no register ever moves between chunks.
// Slow chunks (near the end of a band) mask cells past the diagonal's end:
// cell (column jr + b, diagonal g0 + d) exists iff d < ghi_rel and
// jr + b < min(lim0 - d, ncols).
template <int R, bool FAST, int OFF, bool GROUP>
__device__ __forceinline__ void chunk_fp32(const char* rbase, const char* cbuf,
                                           DenseWin (&win)[R / 2], float2 (&nc2)[R / 2],
                                           float (&acc)[2 * R], const unsigned (&tag)[R],
                                           int lim0, int ncols, int ghi_rel, int jr, int lane,
                                           int& colkey) {
    constexpr int H = R / 2;
    static_assert(R % 2 == 0, "columns are processed in pairs");
    const float2 one2 = make_float2(1.f, 1.f);
    // Columns go in pairs (b, b + 1): row slot s = b + d takes cell d of
    // column b and cell d - 1 of column b + 1, so one 3-input min per slot
    // serves both columns (9 row-min instructions per 2R cells, not 2R).
#pragma unroll
    for (int b = 0; b < R; b += 2) {
        float kb[R];  // column b's tagged cells, by diagonal
        {
            {
                // record tbase + b + H - 1; tbase % 8 == 0, so its slot % 8 == H - 1
                const char* p = rbase + rec_step<H - 1>(b);
                win[(b + H - 1) % H].dfdg = *reinterpret_cast<const float4*>(p);
                win[(b + H - 1) % H].nn = *reinterpret_cast<const float2*>(p + 16);
            }
            const float4 cv = *reinterpret_cast<const float4*>(cbuf + 32 * b);
            const float2 cnn = *reinterpret_cast<const float2*>(cbuf + 32 * b + 16);
            float cmin;
#pragma unroll
            for (int a = 0; a < H; ++a) {
                const DenseWin& rv = win[(b + a) % H];
                const float2 nn2 = __fmul2_rn(cnn, rv.nn);
                const float2 u2 = __ffma2_rn(nc2[a], nn2, one2);
                nc2[a] = __ffma2_rn(lo2(cv), hi2(rv.dfdg), nc2[a]);
                nc2[a] = __ffma2_rn(lo2(rv.dfdg), hi2(cv), nc2[a]);
                kb[a] = GROUP ? u2.x : tag_key(u2.x, tag[a]);
                kb[a + H] = GROUP ? u2.y : tag_key(u2.y, tag[a + H]);
                if (!FAST) {
                    const int l0 = a < ghi_rel ? min(lim0 - a, ncols) : 0;
                    const int l1 = a + H < ghi_rel ? min(lim0 - a - H, ncols) : 0;
                    if (jr + b >= l0) kb[a] = kInf;
                    if (jr + b >= l1) kb[a + H] = kInf;
                }
                cmin = a == 0 ? fminf(kb[a], kb[a + H]) : fmin3(cmin, kb[a], kb[a + H]);
            }
            acc[(b + OFF) % (2 * R)] = fminf(acc[(b + OFF) % (2 * R)], kb[0]);
            const int kmin =
                __reduce_min_sync(kFullMask, __float_as_int(GROUP ? tag_lane(cmin, lane) : cmin));
            colkey = (lane == b + OFF) ? kmin : colkey;
        }
        {
            const int c = b + 1;
            {
                const char* p = rbase + rec_step<H - 1>(c);
                win[(c + H - 1) % H].dfdg = *reinterpret_cast<const float4*>(p);
                win[(c + H - 1) % H].nn = *reinterpret_cast<const float2*>(p + 16);
            }
            const float4 cv = *reinterpret_cast<const float4*>(cbuf + 32 * c);
            const float2 cnn = *reinterpret_cast<const float2*>(cbuf + 32 * c + 16);
            float cmin;
#pragma unroll
            for (int a = 0; a < H; ++a) {
                const DenseWin& rv = win[(c + a) % H];
                const float2 nn2 = __fmul2_rn(cnn, rv.nn);
                const float2 u2 = __ffma2_rn(nc2[a], nn2, one2);
                nc2[a] = __ffma2_rn(lo2(cv), hi2(rv.dfdg), nc2[a]);
                nc2[a] = __ffma2_rn(lo2(rv.dfdg), hi2(cv), nc2[a]);
                float k0 = GROUP ? u2.x : tag_key(u2.x, tag[a]);
                float k1 = GROUP ? u2.y : tag_key(u2.y, tag[a + H]);
                if (!FAST) {
                    const int l0 = a < ghi_rel ? min(lim0 - a, ncols) : 0;
                    const int l1 = a + H < ghi_rel ? min(lim0 - a - H, ncols) : 0;
                    if (jr + c >= l0) k0 = kInf;
                    if (jr + c >= l1) k1 = kInf;
                }
                // slot c + a: cell a of column c and cell a + 1 of column b
                acc[(c + a + OFF) % (2 * R)] = fmin3(acc[(c + a + OFF) % (2 * R)], k0, kb[a + 1]);
                // slot c + a + H: cell a + H of column c and cell a + H + 1 of column
                // b.  Slots b + R - 1 and b + R begin new rows here (these are their
                // first cells), so they are assigned and no slot needs a reset.
                if (a == H - 1)
                    acc[(c + a + H + OFF) % (2 * R)] = k1;
                else if (a == H - 2)
                    acc[(c + a + H + OFF) % (2 * R)] = fminf(k1, kb[a + H + 1]);
                else
                    acc[(c + a + H + OFF) % (2 * R)] =
                        fmin3(acc[(c + a + H + OFF) % (2 * R)], k1, kb[a + H + 1]);
                cmin = a == 0 ? fminf(k0, k1) : fmin3(cmin, k0, k1);
            }
            const int kmin =
                __reduce_min_sync(kFullMask, __float_as_int(GROUP ? tag_lane(cmin, lane) : cmin));
            colkey = (lane == c + OFF) ? kmin : colkey;
        }
    }
}

template <int R, bool GROUP>
__device__ void tile_dense(const Fp32TileParams& P, int64_t band, int64_t seg, int lane, float* ring,
                          char* rring, char* cring) {
    constexpr int H = R / 2;
    constexpr int RING = 32 * R;
    const int64_t gb = P.g_lo + band * (int64_t)RING;
    const int64_t g0 = gb + (int64_t)lane * R;
    const int64_t jmax = P.PL - gb;
    const int64_t j0 = seg * P.K;
    const int64_t j1 = min(j0 + P.K, jmax);
    if (j0 >= j1) return;
    // guarded form: tiles touching a hazard window are evaluated in FP64
    if (P.hazard && fp32_tile_hazardous(P, gb, j0, j1, 32 * R)) return;
    const float ulim = (float)(1.0 + 1.0 / (double)P.m);
    const unsigned ulim_ord = ord_f32(ulim);
    // cell (column j, diagonal g0 + d) is evaluated iff d < ghi_rel and
    // j - j0 < min(lim0 - d, ncols); every cell of a chunk ending at or
    // before minlim exists
    const int ncols = (int)(j1 - j0);
    const int lim0 = (int)min(P.PL - g0 - j0, (int64_t)ncols + R);
    const int ghi_rel = (int)max(min(P.g_hi - g0, (int64_t)R), (int64_t)0);
    const int minlim = ghi_rel < R ? 0 : min(lim0 - (R - 1), ncols);
    // tag of cell d: lane << 3 | d
    unsigned tag[R];
#pragma unroll
    for (int a = 0; a < R; ++a) tag[a] = ((unsigned)lane << 3) | (unsigned)a;

    double anchor[R];
    tile_anchor(P, j0, gb, g0, lane, rring, anchor);
    float nc[R];
#pragma unroll
    for (int a = 0; a < R; ++a) nc[a] = (float)anchor[a];
    float2 nc2[H];
#pragma unroll
    for (int a = 0; a < H; ++a) nc2[a] = make_float2(nc[a], nc[a + H]);

    // ---- ring of row partials for this tile -----------------------------------
    for (int k = lane; k < kRowChunks * kRowStride; k += 32) ring[k] = kInf;
    __syncwarp();

    // row partials: row o of chunk c (o in [0, 2R-1)) lives in acc[(o + R*(c%2)) % 2R]
    float acc[2 * R];
#pragma unroll
    for (int k = 0; k < 2 * R; ++k) acc[k] = kInf;

    // row records of the band, tile-relative index t = row - (j0 + gb), staged
    // in the warp's shared-memory ring; before chunk pair i it holds t < fill
    const uint4* rsrc = reinterpret_cast<const uint4*>(
        reinterpret_cast<const RowRec*>(P.rowrec) + (j0 + gb));
    int fill = 33 * R + H;
    for (int i = lane; i < 2 * fill; i += 32) rec_store(rring, i >> 1, i & 1, __ldg(rsrc + i));
    // column records of a chunk pair (2R records), double-buffered
    const uint4* csrc = reinterpret_cast<const uint4*>(
        reinterpret_cast<const RowRec*>(P.colrec) + j0);
    *reinterpret_cast<uint4*>(cring + 16 * lane) = __ldg(csrc + lane);
    __syncwarp();
    DenseWin win[H];
#pragma unroll
    for (int k = 0; k < H - 1; ++k) {
        const char* p = rring + rec_off(rec_slot(lane * R + k));
        win[k].dfdg = *reinterpret_cast<const float4*>(p);
        win[k].nn = *reinterpret_cast<const float2*>(p + 16);
    }

    // Row partials leave the registers through a ring of kRowChunks chunks of
    // R rows in shared memory: row t of the tile sits at
    // ((t / R) % kRowChunks) * kRowStride + t % R.  With 34 chunks the rows
    // finished by lane 0 in a chunk pair stay put until they are flushed at the
    // end of the pair.
    constexpr int RK_CHUNKS = kRowChunks;
    static_assert(R == 8, "row ring stride is laid out for 8 rows per chunk");
    int cb = 0;                              // column buffer of the current pair
    int rslot = rec_slot(lane * R + H - 1);  // record slot of jr + lane*R + H - 1
    int kslot = lane;                        // (jr / R + lane) % RK_CHUNKS
    int jr = 0;
    for (; jr < ncols; jr += 2 * R) {
        // prefetch what the next pair appends, 2R row records (ring slots this
        // pair does not read: the ring holds 33R + H + 2R < kRecRing records
        // from the pair's first) and 2R column records (the other buffer),
        // copied straight into shared memory while the pair runs
        {
            const int s = rec_slot(fill + (lane >> 1));
            const uint4* src = rsrc + 2 * (int64_t)fill + lane;
            cp_async16(rring + rec_off(s) + 16 * (lane & 1), src);
            if (s < kRecMirror) cp_async16(rring + rec_off(s + kRecRing) + 16 * (lane & 1), src);
            cp_async16(cring + (cb ^ 1) * 64 * R + 16 * lane, csrc + 2 * (int64_t)(jr + 2 * R) + lane);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        int colkey = 0x7fffffff;
        const char* cbuf = cring + cb * 64 * R;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int jh = jr + half * R;
            const char* rbase = rring + rec_off(rslot);
            rslot += R;
            if (rslot >= kRecRing) rslot -= kRecRing;
            const bool fast = __all_sync(kFullMask, jh + R <= minlim);
            if (half == 0) {
                if (fast)
                    chunk_fp32<R, true, 0, GROUP>(rbase, cbuf, win, nc2, acc, tag, lim0, ncols, ghi_rel, jh, lane, colkey);
                else
                    chunk_fp32<R, false, 0, GROUP>(rbase, cbuf, win, nc2, acc, tag, lim0, ncols, ghi_rel, jh, lane, colkey);
            } else {
                if (fast)
                    chunk_fp32<R, true, R, GROUP>(rbase, cbuf + 32 * R, win, nc2, acc, tag, lim0,
                                           ncols, ghi_rel, jh, lane, colkey);
                else
                    chunk_fp32<R, false, R, GROUP>(rbase, cbuf + 32 * R, win, nc2, acc, tag,
                                            lim0, ncols, ghi_rel, jh, lane, colkey);
            }
            // this chunk's lower half (rows jh + g0 + [0, R)) is final for the lane
            const int ks = (kslot + half) >= RK_CHUNKS ? kslot + half - RK_CHUNKS : kslot + half;
            float4* rv4 = reinterpret_cast<float4*>(ring + ks * kRowStride);
#pragma unroll
            for (int v = 0; v < R / 4; ++v) {
                float4 t = rv4[v];
                t.x = fminf(t.x, lane_min<GROUP>(acc[(4 * v + 0 + half * R) % (2 * R)], lane));
                t.y = fminf(t.y, lane_min<GROUP>(acc[(4 * v + 1 + half * R) % (2 * R)], lane));
                t.z = fminf(t.z, lane_min<GROUP>(acc[(4 * v + 2 + half * R) % (2 * R)], lane));
                t.w = fminf(t.w, lane_min<GROUP>(acc[(4 * v + 3 + half * R) % (2 * R)], lane));
                rv4[v] = t;
            }
            // lane l's next merge reads the chunk lane l + 1 has just written
            __syncwarp();
        }
        kslot += 2;
        if (kslot >= RK_CHUNKS) kslot -= RK_CHUNKS;
        __syncwarp();
        // columns jr + [0, 2R): one per lane
        if (lane < 2 * R) {
            if constexpr (GROUP) {
                // rows jr + [0, 2R) of the tile have met every lane: flush, free
                const int c = jr / R + (lane >> 3);
                const int e = (c % RK_CHUNKS) * kRowStride + (lane & (R - 1));
                const float v = ring[e];
                ring[e] = kInf;
                const int64_t j = j0 + jr + lane, r = j0 + gb + jr + lane;
                flush_col_group(P, (unsigned)colkey, j, gb, ulim_ord);
                flush_row_group(P, v, r, gb, ulim_ord);
            } else {
                const unsigned bits = (unsigned)colkey;
                const float u = untag_value(bits);
                if (u < ulim) {
                    const unsigned t = bits & kTagMask;
                    const int64_t j = j0 + jr + lane;
                    const int64_t q = j + gb + (int64_t)(t >> 3) * R + (t & 7u);
                    atomicMin(P.key + j, ((unsigned long long)ord_f32(u) << 32) | (unsigned long long)q);
                }
                // rows jr + [0, 2R) of the tile have met every lane: flush, free
                const int c = jr / R + (lane >> 3);
                const int e = (c % RK_CHUNKS) * kRowStride + (lane & (R - 1));
                const float v = ring[e];
                ring[e] = kInf;
                flush_row(P, v, j0 + gb + jr + lane, gb, ulim);
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        cb ^= 1;
        fill += 2 * R;
        __syncwarp();
    }

    // drain: the carried upper half (rows jr + lane*R + [0, R-1)), then every slot
    {
        float* base = ring + kslot * kRowStride;
#pragma unroll
        for (int k = 0; k < R - 1; ++k) base[k] = fminf(base[k], lane_min<GROUP>(acc[k], lane));
    }
    __syncwarp();
    const int cend = jr / R;
    for (int e = lane; e < RK_CHUNKS * R; e += 32) {
        const int cs = e / R;
        const int rel = (cs - cend % RK_CHUNKS + RK_CHUNKS) % RK_CHUNKS;
        const int64_t r = j0 + gb + (int64_t)(cend + rel) * R + (e % R);
        if constexpr (GROUP)
            flush_row_group(P, ring[cs * kRowStride + e % R], r, gb, ulim_ord);
        else
            flush_row(P, ring[cs * kRowStride + e % R], r, gb, ulim);
    }
    __syncwarp();
}

constexpr int kDenseSmem = kRecRingBytes + kRowChunks * kRowStride * (int)sizeof(float) + 4 * 32 * kR;
static_assert(kDenseSmem % 16 == 0, "warps' areas stay 16-byte aligned");

// ---- passes behind the gate ---------------------------------------------------
constexpr int kPassCols = 16;    // columns per pass
constexpr int kGroups = 40;  // ring: groups of 8 rows; a pass reads 34, 2 more arrive
constexpr int kPad = 9;      // elements between groups: lanes 8 rows apart hit distinct banks
// The gate asks for nc * nn_r < -sn / nn_j with sn = 1 - bound - kGateSlack, where u
// = fl(1 + nc * fl(nn_j nn_r)) <= bound is meant: roundings of four values below
// 1.01 in size near a bound, 2.5e-7 together (5e-7 where nn_j nn_r is subnormal).
constexpr float kGateSlack = 2e-6f;
constexpr int kTileSmem = kGroups * kPad * 12 + 2 * kPassCols * 16 +
                          2 * kGroups * kRowStride * 4 + 2 * kPassCols * 4 + kGroups * 4;
static_assert(kTileSmem % 16 == 0, "warps' areas stay 16-byte aligned");
static_assert(kAnchorBytes <= kTileSmem, "anchor staging fits");
__device__ __forceinline__ int wrap_group(int s) { return s < kGroups ? s : s - kGroups; }

// High word of a key as it stands (merged meanwhile by other warps).
__device__ __forceinline__ unsigned ld_key_hi(const unsigned long long* key) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];"
                 : "=r"(v)
                 : "l"(reinterpret_cast<const unsigned*>(key) + 1));
    return v;
}
// Where a row starts.
__device__ __forceinline__ unsigned key_bound(unsigned hi) { return fp32_key_bound(hi, true); }

// The warp's shared memory for a tile.
struct TileSmem {
    float2* dd;      // row terms df, dg, kPad per group
    float* nn;       // ... and nn
    float4* col;     // column terms -df, -dg, nn, 1 / nn, two buffers of kPassCols
    float* best;     // best tagged distance per row, kRowStride per group
    float* start;    // what it started from
    unsigned* cthr;  // column bounds (bit patterns), two buffers of kPassCols
    unsigned* gate;  // per group: the loosest of its rows' bests (bit pattern)
    __device__ __forceinline__ explicit TileSmem(char* p) {
        col = reinterpret_cast<float4*>(p);
        best = reinterpret_cast<float*>(col + 2 * kPassCols);
        start = best + kGroups * kRowStride;
        dd = reinterpret_cast<float2*>(start + kGroups * kRowStride);
        nn = reinterpret_cast<float*>(dd + kGroups * kPad);
        cthr = reinterpret_cast<unsigned*>(nn + kGroups * kPad);
        gate = cthr + 2 * kPassCols;
    }
    // Copies the terms of 16 rows (two groups from slot s) from pair records.
    __device__ __forceinline__ void stage_rows(int s, const float* src, int lane) const {
        const int e = (s + ((lane & 15) >> 3)) * kPad + (lane & 7);
        const float* r = src + kRecFloats * (lane & 15);
        cp_async4(reinterpret_cast<float*>(dd + e) + (lane >> 4), r + 2 * (lane >> 4));
        if (lane < 16) cp_async4(nn + e, r + 4);
    }
    // ... and of kPassCols columns into buffer b
    __device__ __forceinline__ void stage_cols(int b, const float* src, int lane) const {
        float* d = reinterpret_cast<float*>(col + b * kPassCols);
        const float* r = src + kRecFloats * (lane >> 1) + 4 * (lane & 1);
        cp_async4(d + 4 * (lane >> 1) + 2 * (lane & 1), r);
        cp_async4(d + 4 * (lane >> 1) + 2 * (lane & 1) + 1, r + 2);
    }
    __device__ __forceinline__ unsigned group_gate(int s) const {
        const float4 a = *reinterpret_cast<const float4*>(best + s * kRowStride);
        const float4 b = *reinterpret_cast<const float4*>(best + s * kRowStride + 4);
        const float m = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)),
                              fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        return __float_as_uint(fmaxf(m, 0.f));
    }
};

// A lane's window of 8 rows.
struct RowWin {
    float df[8], dg[8], nn[8];
    __device__ __forceinline__ void load(const TileSmem& sm, int s) {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const float2 x = sm.dd[s * kPad + a];
            df[a] = x.x;
            dg[a] = x.y;
            nn[a] = sm.nn[s * kPad + a];
        }
    }
};

__device__ __forceinline__ unsigned gate_pass(const TileSmem& sm, int s1, int s2, const float4* col,
                                           float sn, RowWin& win, float (&nc)[8]) {
    const float2* d = sm.dd + s1 * kPad;
    const float* n = sm.nn + s1 * kPad;
    unsigned t = 0;
#pragma unroll 1
    for (int h = 0; h < kPassCols / 8; ++h) {
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const float4 cv = col[b];
            const float c = sn * cv.w;
            float v[8];
#pragma unroll
            for (int a = 0; a < 8; ++a) v[a] = __fmaf_rn(nc[a], win.nn[(b + a) % 8], c);
#pragma unroll
            for (int a = 0; a < 8; ++a) nc[a] = __fmaf_rn(cv.x, win.dg[(b + a) % 8], nc[a]);
#pragma unroll
            for (int a = 0; a < 8; ++a) nc[a] = __fmaf_rn(cv.y, win.df[(b + a) % 8], nc[a]);
            {  // row b gives way to row b + 8
                const float2 x = d[b];
                win.df[b] = x.x;
                win.dg[b] = x.y;
                win.nn[b] = n[b];
            }
#pragma unroll
            for (int a = 0; a < 8; a += 2) t |= __float_as_uint(v[a]) | __float_as_uint(v[a + 1]);
        }
        d = sm.dd + s2 * kPad;
        n = sm.nn + s2 * kPad;
        col += 8;
    }
    return t;
}

// One pass with the selection.  Columns go in pairs: row element e takes cell
// e - b of column b and cell e - b - 1 of column b + 1, so one 3-input minimum per
// element serves both; a column's minimum over the warp is one REDUX, kept by lane
// b in colkey.  Elements 8g .. 8g + 7 go to the lane's group g once 8 columns have
// met them.  EDGE: cell (column jr + b, diagonal g0 + d) exists iff d < ghi_rel and
// jr + b < min(lim0 - d, ncols).  Window as in gate_pass.  Returns whether a row's
// best fell.
template <bool EDGE, bool GROUP>
__device__ __forceinline__ bool dense_pass(const TileSmem& sm, int s0, int s1, int s2,
                                           const float4* col, RowWin& win, float (&nc)[8], int lim0,
                                           int ncols, int ghi_rel, int jr, int lane, int& colkey) {
    const float2* rd = sm.dd + s1 * kPad;
    const float* rn = sm.nn + s1 * kPad;
    float acc[16];  // row elements 8h .. 8h + 15
    unsigned fell = 0;
    int sg = s0;  // group of the first 8
    auto merge = [&]() {
        __syncwarp();  // lane l's group g + 1 is lane l + 1's group g
        float4* e = reinterpret_cast<float4*>(sm.best + sg * kRowStride);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 o = e[h];
            float4 v;
            const float* k = acc + 4 * h;
            v.x = fminf(o.x, lane_min<GROUP>(k[0], lane));
            v.y = fminf(o.y, lane_min<GROUP>(k[1], lane));
            v.z = fminf(o.z, lane_min<GROUP>(k[2], lane));
            v.w = fminf(o.w, lane_min<GROUP>(k[3], lane));
            e[h] = v;
            fell |= __float_as_uint(v.x) ^ __float_as_uint(o.x);
            fell |= __float_as_uint(v.y) ^ __float_as_uint(o.y);
            fell |= __float_as_uint(v.z) ^ __float_as_uint(o.z);
            fell |= __float_as_uint(v.w) ^ __float_as_uint(o.w);
        }
    };
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = kInf;
#pragma unroll 1
    for (int h = 0; h < kPassCols / 8; ++h) {
#pragma unroll
        for (int b = 0; b < 8; b += 2) {
            float kb[8];  // column b's cells
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c = b + i;
                const float4 cv = col[c];
                float kc[8], cmin = kInf;
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                    const int w = (c + d) % 8;
                    const float u = __fmaf_rn(nc[d], __fmul_rn(cv.z, win.nn[w]), 1.f);
                    nc[d] = __fmaf_rn(cv.x, win.dg[w], nc[d]);
                    nc[d] = __fmaf_rn(win.df[w], cv.y, nc[d]);
                    kc[d] = GROUP ? u : tag_key(u, ((unsigned)lane << 3) | (unsigned)d);
                    if (EDGE) {
                        const int l = d < ghi_rel ? min(lim0 - d, ncols) : 0;
                        if (jr + c >= l) kc[d] = kInf;
                    }
                    if (d % 2) cmin = d == 1 ? fminf(kc[0], kc[1]) : fmin3(cmin, kc[d - 1], kc[d]);
                }
                {  // row c gives way to row c + 8
                    const float2 x = rd[c];
                    win.df[c] = x.x;
                    win.dg[c] = x.y;
                    win.nn[c] = rn[c];
                }
                const int kmin =
                    __reduce_min_sync(kFullMask, __float_as_int(GROUP ? tag_lane(cmin, lane) : cmin));
                colkey = lane == 8 * h + c ? kmin : colkey;
                if (i == 0) {
#pragma unroll
                    for (int d = 0; d < 8; ++d) kb[d] = kc[d];
                    continue;
                }
                acc[b] = fminf(acc[b], kb[0]);
#pragma unroll
                for (int d = 0; d < 7; ++d) {
                    const int e = b + 1 + d;  // first met by column b when d == 6
                    acc[e] = d == 6 ? fminf(kb[d + 1], kc[d]) : fmin3(acc[e], kb[d + 1], kc[d]);
                }
                acc[b + 8] = kc[7];
            }
        }
        merge();
#pragma unroll
        for (int k = 0; k < 7; ++k) acc[k] = acc[k + 8];
        acc[7] = kInf;  // no cell yet
        sg = h == 0 ? s1 : s2;
        rd = sm.dd + s2 * kPad;
        rn = sm.nn + s2 * kPad;
        col += 8;
        jr += 8;
    }
    merge();
    return __any_sync(kFullMask, fell != 0);
}

template <bool GROUP>
__device__ void tile_gate(const Fp32TileParams& P, int64_t band, int64_t seg, int lane,
                          const TileSmem& sm) {
    constexpr int R = kR;
    const int64_t gb = P.g_lo + band * (int64_t)(32 * R);
    const int64_t g0 = gb + (int64_t)lane * R;
    const int64_t jmax = P.PL - gb;
    const int64_t j0 = seg * P.K;
    const int64_t j1 = min(j0 + P.K, jmax);
    if (j0 >= j1) return;
    // guarded form: tiles touching a hazard window are evaluated in FP64
    if (P.hazard && fp32_tile_hazardous(P, gb, j0, j1, 32 * R)) return;
    const float ulim = (float)(1.0 + 1.0 / (double)P.m);
    const unsigned ulim_ord = ord_f32(ulim);
    // extents of the tile's cells, as in tile_dense
    const int ncols = (int)(j1 - j0);
    const int lim0 = (int)min(P.PL - g0 - j0, (int64_t)ncols + R);
    const int ghi_rel = (int)max(min(P.g_hi - g0, (int64_t)R), (int64_t)0);
    const int minlim = __reduce_min_sync(kFullMask, ghi_rel < R ? 0 : min(lim0 - (R - 1), ncols));

    double anchor[R];
    tile_anchor(P, j0, gb, g0, lane, reinterpret_cast<char*>(sm.col), anchor);
    float nc[R];
#pragma unroll
    for (int a = 0; a < R; ++a) nc[a] = (float)anchor[a];

    // groups 0 .. 33 and the first pass's columns; from here on lanes 0 - 15 look
    // after rows, lanes 16 - 31 after columns
    const int64_t rb = j0 + gb;  // row of element 0 of group 0
    const float* nrow = fp32_record(reinterpret_cast<const float*>(P.rowrec), rb);
    const float* ncol = fp32_record(reinterpret_cast<const float*>(P.colrec), j0);
    for (int i = 0; i < 17; ++i) sm.stage_rows(2 * i, fp32_record(nrow, 16 * i), lane);
    sm.stage_cols(0, ncol, lane);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int i = lane; i < 34 * R; i += 32) {
        const unsigned f = rb + i < P.PL ? key_bound(ld_key_hi(P.key + rb + i)) : 0u;
        const int e = (i / R) * kRowStride + i % R;
        sm.best[e] = __uint_as_float(f);
        sm.start[e] = __uint_as_float(f);
    }
    unsigned cgate = 0;
    if (lane < kPassCols) {
        cgate = j0 + lane < P.PL ? key_bound(ld_key_hi(P.key + j0 + lane)) : 0u;
        sm.cthr[lane] = cgate | kTagMask;
    }
    cgate = __reduce_max_sync(kFullMask, cgate);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    sm.gate[lane] = sm.group_gate(lane);
    if (lane < 2) sm.gate[32 + lane] = sm.group_gate(32 + lane);
    __syncwarp();
    RowWin win;
    win.load(sm, lane);

    const int64_t inc0 = lane < 16 ? rb + 34 * R + lane : j0 + lane;  // - 16 + kPassCols
    int s0 = lane;  // slot of the lane's first group
    int sf = 0;     // slot of the first group that the pass finishes
    int cb = 0;
    bool sel = false;
    int skip = 0, streak = 0;
    int jr = 0;
    for (; jr < ncols; jr += kPassCols) {
        // what the next pass appends: 16 rows, 16 columns and their keys
        const int sn = wrap_group(sf + 34);
        sm.stage_rows(sn, fp32_record(nrow, 34 * R + (int64_t)jr), lane);
        sm.stage_cols(cb ^ 1, fp32_record(ncol, jr + kPassCols), lane);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const int64_t inc = inc0 + jr;
        unsigned f = 0;
        if (inc < P.PL) f = ld_key_hi(P.key + inc);

        const int s1 = wrap_group(s0 + 1), s2 = wrap_group(s0 + 2);
        const float bound =
            __uint_as_float(max(max(sm.gate[s0], sm.gate[s1]), max(sm.gate[s2], cgate)) | kTagMask);
        const float4* col = sm.col + cb * kPassCols;
        const unsigned* cthr = sm.cthr + cb * kPassCols;
        const bool inside = jr + kPassCols <= minlim;
        // A pass after one that lowered something goes straight on; so do the next
        // 1, 2, 4 .. 16 passes after gates that opened in a row, where a gate in
        // every pass would only add to the selection.
        bool open = !inside || sel || skip > 0;
        skip -= skip > 0;
        const bool again = !open;
        if (!open) {
            float q0[8];
#pragma unroll
            for (int a = 0; a < 8; ++a) q0[a] = nc[a];
            const float sn = (1.f - bound) - kGateSlack;
            const unsigned t = gate_pass(sm, s1, s2, col, sn, win, nc);
            open = __any_sync(kFullMask, (int)t < 0 || sn <= 0.f);
            streak = open ? min(max(2 * streak, 1), 16) : 0;
            skip = streak;
            if (open) {
#pragma unroll
                for (int a = 0; a < 8; ++a) nc[a] = q0[a];
            }
        }
        sel = false;
        if (open) {
            if (again) win.load(sm, s0);
            int colkey = 0x7fffffff;
            sel = inside ? dense_pass<false, GROUP>(sm, s0, s1, s2, col, win, nc, lim0, ncols, ghi_rel, jr,
                                                    lane, colkey)
                         : dense_pass<true, GROUP>(sm, s0, s1, s2, col, win, nc, lim0, ncols, ghi_rel, jr,
                                                   lane, colkey);
            // columns jr + lane at or below their keys
            bool low = false;
            if (lane < kPassCols) {
                const float v = untag_value((unsigned)colkey);
                low = v <= __uint_as_float(cthr[lane]);
                const int64_t j = j0 + jr + lane;
                if (low) {
                    if constexpr (GROUP) {
                        flush_col_group(P, (unsigned)colkey, j, gb, ulim_ord);
                    } else if (v < ulim) {
                        atomicMin(P.key + j, ((unsigned long long)ord_f32(v) << 32) |
                                                 (unsigned long long)(j + gb + ((unsigned)colkey & kTagMask)));
                    }
                }
            }
            sel |= __any_sync(kFullMask, low);
        }
        __syncwarp();
        // the pass's first two groups have met every lane: merge the rows that fell
        f = inc < P.PL ? key_bound(f) : 0u;
        if (lane < 16) {
            const int e = (sf + (lane >> 3)) * kRowStride + (lane & 7);
            const float v = sm.best[e];
            if (v < sm.start[e]) {
                if constexpr (GROUP)
                    flush_row_group(P, v, rb + jr + lane, gb, ulim_ord);
                else
                    flush_row(P, v, rb + jr + lane, gb, ulim);
            }
            const int en = (sn + (lane >> 3)) * kRowStride + (lane & 7);
            sm.best[en] = __uint_as_float(f);
            sm.start[en] = __uint_as_float(f);
        } else {
            sm.cthr[(cb ^ 1) * kPassCols + lane - 16] = f | kTagMask;
        }
        const unsigned g0v = __reduce_max_sync(kFullMask, lane < 8 ? f : 0u);
        const unsigned g1v = __reduce_max_sync(kFullMask, (lane & 24) == 8 ? f : 0u);
        cgate = __reduce_max_sync(kFullMask, lane >= 16 ? f : 0u);
        if (lane == 0) {
            sm.gate[sn] = g0v;
            sm.gate[sn + 1] = g1v;
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
        const int e = wrap_group(sf + i / R) * kRowStride + i % R;
        const float v = sm.best[e];
        if (v < sm.start[e]) {
            if constexpr (GROUP)
                flush_row_group(P, v, rb + jr + i, gb, ulim_ord);
            else
                flush_row(P, v, rb + jr + i, gb, ulim);
        }
    }
    __syncwarp();
}

constexpr int kFp32WarpsPerBlock = 4;
// CTAs per SM: the gate's registers allow 4 (n = 1,048,576: 127 ms against 134 at
// 3), the dense way's 3 (178 ms against 185), except with group keys, which need
// no per-cell tags.
template <Fp32Way WAY, bool GROUP>
constexpr int fp32_blocks_per_sm() {
    return WAY == kFp32Gate || (WAY == kFp32Dense && GROUP) ? 4 : 3;
}
template <Fp32Way WAY>
struct Fp32Smem {
    static constexpr int kPerWarp =
        WAY == kFp32Gate ? kTileSmem : (kDenseSmem > kTileSmem ? kDenseSmem : kTileSmem);
    static constexpr int kPerBlock = kFp32WarpsPerBlock * kPerWarp;
};

template <Fp32Way WAY, bool GROUP>
__global__ void __launch_bounds__(32 * kFp32WarpsPerBlock, fp32_blocks_per_sm<WAY, GROUP>())
    fp32_join_kernel(const Fp32TileParams* __restrict__ series, int nseries, int64_t total,
                     unsigned long long* __restrict__ counter) {
    extern __shared__ __align__(128) char smem_fp32[];
    const int lane = threadIdx.x & 31;
    char* mine = smem_fp32 + (threadIdx.x >> 5) * Fp32Smem<WAY>::kPerWarp;
    for_each_tile(series, nseries, total, counter, lane,
                  [&](const Fp32TileParams& P, int64_t band, int64_t seg) {
                      if (WAY == kFp32Gate || (WAY == kFp32Mixed && fp32_gate_pays(P.m, P.PL)))
                          tile_gate<GROUP>(P, band, seg, lane, TileSmem(mine));
                      else
                          tile_dense<kR, GROUP>(P, band, seg, lane, reinterpret_cast<float*>(mine + kRecRingBytes),
                                                mine, mine + kRecRingBytes + kRowChunks * kRowStride * 4);
                  });
}

template <Fp32Way WAY, bool GROUP>
void launch_way(const Fp32TileParams* series, int nseries, int64_t total, unsigned long long* counter,
                cudaStream_t s) {
    const int64_t want = (total + kFp32WarpsPerBlock - 1) / kFp32WarpsPerBlock;
    const int64_t blocks = std::min<int64_t>(want, (int64_t)sm_count() * fp32_blocks_per_sm<WAY, GROUP>());
    if (blocks > 0)
        fp32_join_kernel<WAY, GROUP><<<(unsigned)blocks, 32 * kFp32WarpsPerBlock, Fp32Smem<WAY>::kPerBlock, s>>>(
            series, nseries, total, counter);
}

}  // namespace

void fp32_tile_plan(int64_t PL, int64_t g_lo, int64_t g_hi, int64_t K, int R, int64_t& nbands,
                    int64_t& seg_per_pair, int64_t& ntiles) {
    const int64_t span = 32 * R;
    const int64_t ndiag = g_hi > g_lo ? g_hi - g_lo : 0;
    nbands = (ndiag + span - 1) / span;
    const int64_t npairs = (nbands + 1) / 2;
    int64_t spp = 0;
    for (int64_t p = 0; p < npairs; ++p) {
        int64_t t = (PL - (g_lo + p * span) + K - 1) / K;
        const int64_t p2 = nbands - 1 - p;
        if (p2 > p) t += (PL - (g_lo + p2 * span) + K - 1) / K;
        spp = std::max(spp, t);
    }
    seg_per_pair = std::max<int64_t>(spp, 1);
    ntiles = npairs * seg_per_pair;
}

template <int R>
void configure_fp32_join() {
    static_assert(R == kR, "the tile kernel is laid out for 8 diagonals per lane");
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(fp32_join_kernel<kFp32Dense, false>, attr, Fp32Smem<kFp32Dense>::kPerBlock);
    cudaFuncSetAttribute(fp32_join_kernel<kFp32Dense, true>, attr, Fp32Smem<kFp32Dense>::kPerBlock);
    cudaFuncSetAttribute(fp32_join_kernel<kFp32Gate, false>, attr, Fp32Smem<kFp32Gate>::kPerBlock);
    cudaFuncSetAttribute(fp32_join_kernel<kFp32Gate, true>, attr, Fp32Smem<kFp32Gate>::kPerBlock);
    cudaFuncSetAttribute(fp32_join_kernel<kFp32Mixed, false>, attr, Fp32Smem<kFp32Mixed>::kPerBlock);
}

template <int R>
void launch_fp32_join(const Fp32TileParams* series_dev, int nseries, int64_t total,
                      unsigned long long* counter, cudaStream_t s, Fp32Way way, bool group) {
    // the shared-memory limit is a per-device attribute; setting it is
    // idempotent, so concurrent first launches (server threads) are harmless
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        configure_fp32_join<R>();
        configured.fetch_or(bit, std::memory_order_release);
    }
    if (way == kFp32Mixed)
        launch_way<kFp32Mixed, false>(series_dev, nseries, total, counter, s);
    else if (way == kFp32Gate)
        group ? launch_way<kFp32Gate, true>(series_dev, nseries, total, counter, s)
              : launch_way<kFp32Gate, false>(series_dev, nseries, total, counter, s);
    else
        group ? launch_way<kFp32Dense, true>(series_dev, nseries, total, counter, s)
              : launch_way<kFp32Dense, false>(series_dev, nseries, total, counter, s);
}

template void launch_fp32_join<8>(const Fp32TileParams*, int, int64_t, unsigned long long*,
                                  cudaStream_t, Fp32Way, bool);
template void configure_fp32_join<8>();

}  // namespace mpgpu
