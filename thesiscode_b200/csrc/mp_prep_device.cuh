// Device helpers shared by the single-series and batched preparation kernels.
#pragma once

#include "mp_common.cuh"

namespace mpgpu {

// cs[i] = A[i] + cs[i-1], cs2[i] = A[i]*A[i] + cs2[i-1] in index order
// (ScrimpSequOpt.cpp:43-49).  Each chain is inherently serial, 8 cycles per
// addition (4.3 ms for n = 1M), so one lane of warp 0 and one of warp 1 do nothing
// else, out of shared memory and 16 values ahead: the block's other warps load the
// next chunk of A, square it and write the previous chunk's sums back (all coalesced)
// meanwhile.  n = 1,048,576: 5.4 ms; 8.8 with both chains on two lanes of one
// warp, which squared and selected between the additions.  prefix_block is the work of
// one block of at least 96 threads, C elements per chunk (a multiple of 16).
__device__ __forceinline__ double prefix_chain(const double* src, double* dst, int cnt, double acc) {
    constexpr int U = 16;
    double2 v[U / 2];
    int k = 0;
    if (cnt >= U) {
#pragma unroll
        for (int i = 0; i < U / 2; ++i) v[i] = reinterpret_cast<const double2*>(src)[i];
    }
    for (; k + U <= cnt; k += U) {
        // values of the next round (past the chunk: read from the array's padding, unused)
        double2 w[U / 2];
#pragma unroll
        for (int i = 0; i < U / 2; ++i) {
            const double2 x = v[i];
            w[i] = reinterpret_cast<const double2*>(src + k + U)[i];
            double2 o;
            o.x = __dadd_rn(x.x, acc);
            o.y = __dadd_rn(x.y, o.x);
            acc = o.y;
            reinterpret_cast<double2*>(dst + k)[i] = o;
        }
#pragma unroll
        for (int i = 0; i < U / 2; ++i) v[i] = w[i];
    }
    for (; k < cnt; ++k) {
        acc = __dadd_rn(src[k], acc);
        dst[k] = acc;
    }
    return acc;
}
template <int C>
struct PrefixSmem {
    static constexpr int kBytes = 8 * (4 * (C + 16) + 4 * C);
};
template <int C>
__device__ __forceinline__ void prefix_block(const double* __restrict__ A, int64_t n,
                                             double* __restrict__ cs, double* __restrict__ cs2, char* buf) {
    // [chain][buffer][k]: chain 0 takes A, chain 1 takes A*A
    auto in = reinterpret_cast<double(*)[2][C + 16]>(buf);
    auto out = reinterpret_cast<double(*)[2][C]>(buf + 8 * 4 * (C + 16));
    const int t = threadIdx.x;
    const int64_t nch = (n + C - 1) / C;
    for (int k = t; k < C; k += blockDim.x) {
        const double a = k < n ? A[k] : 0.0;
        in[0][0][k] = a;
        in[1][0][k] = __dmul_rn(a, a);
    }
    __syncthreads();
    double acc = 0.0;
    for (int64_t c = 0; c < nch; ++c) {
        const int b = (int)(c & 1);
        const int cnt = (int)min((int64_t)C, n - c * C);
        if (t < 64) {
            if ((t & 31) == 0) {
                const int h = t >> 5;
                if (c == 0) {  // the first sum is the first value itself
                    acc = in[h][0][0];
                    out[h][0][0] = acc;
                    int k = 1;
                    for (; k < cnt && k < 16; ++k) {
                        acc = __dadd_rn(in[h][0][k], acc);
                        out[h][0][k] = acc;
                    }
                    if (cnt > 16) acc = prefix_chain(in[h][0] + 16, out[h][0] + 16, cnt - 16, acc);
                } else {
                    acc = prefix_chain(in[h][b], out[h][b], cnt, acc);
                }
            }
        } else {
            const int tt = t - 64, nt = blockDim.x - 64;
            if (c + 1 < nch)
                for (int k = tt; k < C; k += nt) {
                    const int64_t i = (c + 1) * C + k;
                    const double a = i < n ? A[i] : 0.0;
                    in[0][b ^ 1][k] = a;
                    in[1][b ^ 1][k] = __dmul_rn(a, a);
                }
            if (c >= 1)
                for (int k = tt; k < C; k += nt) {
                    const int64_t i = (c - 1) * C + k;
                    cs[i] = out[0][b ^ 1][k];
                    cs2[i] = out[1][b ^ 1][k];
                }
        }
        __syncthreads();
    }
    const int64_t c = nch - 1;
    for (int k = t; k < C; k += blockDim.x) {
        const int64_t i = c * C + k;
        if (i < n) {
            cs[i] = out[0][c & 1][k];
            cs2[i] = out[1][c & 1][k];
        }
    }
}

// Welford over the chunk `t` of `chunk` consecutive windows: a full Welford
// pass for the chunk's first window, then the sliding update
//   mean' = mean + (x_in - x_out)/m
//   M2'   = M2 + (x_in - x_out)*(x_in - mean' + x_out - mean).
// Writes mean (FP64) and norm = 1/sqrt(M2) (FP64; NaN for a window whose
// values are all equal -- nchg counts value changes -- so every correlation
// with it is NaN, the reference's zero-variance convention).
__device__ __forceinline__ void welford_chunk(const double* __restrict__ A, int64_t m, int64_t PL,
                                              int64_t chunk, int64_t t, const int* __restrict__ nchg,
                                              double* __restrict__ mean_out,
                                              double* __restrict__ norm_out) {
    const int64_t i0 = t * chunk;
    const int64_t i1 = min(PL, i0 + chunk);
    double mean = 0.0, M2 = 0.0;
    for (int64_t k = 0; k < m; ++k) {
        const double x = A[i0 + k];
        const double delta = x - mean;
        mean += delta / (double)(k + 1);
        M2 += delta * (x - mean);
    }
    const double inv_m = 1.0 / (double)m;
    for (int64_t i = i0; i < i1; ++i) {
        if (i > i0) {
            const double xin = A[i + m - 1], xout = A[i - 1];
            const double mnew = mean + (xin - xout) * inv_m;
            M2 += (xin - xout) * (xin - mnew + xout - mean);
            mean = mnew;
        }
        const bool flat = (nchg[i + m - 1] - nchg[i]) == 0;
        mean_out[i] = mean;
        norm_out[i] = (flat || !(M2 > 0.0)) ? __longlong_as_double(0x7ff8000000000000ll)
                                            : 1.0 / sqrt(M2);
    }
}

// The same statistics for 32 chunks of kStatChunk windows by one block of
// kStatThreads threads, windows base .. base + 32 * kStatChunk - 1 (those below PL).
//
// A chunk is a dependent chain -- a subtraction, a division and an addition per
// sample of its first window, two fused operations per window after it -- so a lane
// of warp 0 runs each, out of shared memory: the block loads its stretch of the
// series coalesced, and warps 1 - 7 turn the second moments into inverse norms and
// write both out while warp 0 walks on.  The division by the sample count b uses the
// correctly rounded 1/b (warp-wide, 32 counts at a time): q = RN(a r) is within 1.5
// units in the last place of a/b, a - b q is exact in one fused operation, and
// RN(q + r (a - b q)) is the correctly rounded quotient (Markstein 1990), because
// with b an integer a/b stays 1/(2b) of a unit away from every rounding boundary.
// Outside the exponents where that holds the division itself is used; 0 / b is 0 either way
// (its sign, which the mean it is added to does not take on, may differ), and has to be
// quick: lanes past the profile's end walk zeros (n = 5,000, m = 1200: 0.55 ms a call with
// the division for them, 0.25 without).
// A window is flat when the last change of value up to its end lies at or before its
// start: a running maximum over the block's stretch in place of counts over the
// whole series.
// n = 65,536, m = 400: 20 us, from 340 us for one thread per chunk reading the series
// from global memory and four launches to count value changes.
constexpr int kStatChunk = 256;
constexpr int kStatThreads = 256;
constexpr int kStatSpan = 32 * kStatChunk;
constexpr int64_t kStatMaxM = 8192;  // longest window whose stretch fits shared memory
constexpr int kStatBatch = 32 * 33;  // 32 windows of 32 chunks, padded
__host__ __device__ constexpr size_t stat_smem_bytes(int64_t m) {
    const size_t S = (size_t)(kStatSpan + m);
    return 8 * (S + S / 256 + 1) + 4 * 8 * kStatBatch + (2 * S + 7) / 8 * 8;
}
// Out of line, so that the chain does not carry a division along.
static __device__ __noinline__ double plain_division(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double quotient(double a, double b, double r) {
    const double q = __dmul_rn(a, r);
    const double z = __fma_rn(__fma_rn(-b, q, a), r, q);
    const double x = fabs(a);
    if ((x <= 1e-280 && x != 0.0) || x >= 1e280) return plain_division(a, b);
    return z;  // NaN, too
}
__device__ __forceinline__ void stat_block(const double* __restrict__ A, int64_t m, int64_t PL, int64_t base,
                                           double* __restrict__ mean_out, double* __restrict__ norm_out,
                                           char* smem) {
    const int S = kStatSpan + (int)m;
    double* sA = reinterpret_cast<double*>(smem);  // element p at p + p / 256
    double* buf = sA + S + S / 256 + 1;            // two batches of means and second moments
    unsigned short* last = reinterpret_cast<unsigned short*>(buf + 4 * kStatBatch);
    __shared__ int wmax[kStatThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int64_t left = PL + m - 1 - base;
    for (int p = tid; p < S; p += kStatThreads) sA[p + (p >> 8)] = p < left ? A[base + p] : 0.0;
    __syncthreads();
    // last[p]: the last q <= p whose value differs from the one before it (0: none)
    {
        const int per = (S + kStatThreads - 1) / kStatThreads;
        const int lo = tid * per, hi = min(S, lo + per);
        auto changed = [&](int p) { return p > 0 && sA[p + (p >> 8)] != sA[p - 1 + ((p - 1) >> 8)]; };
        int mx = 0;
        for (int p = lo; p < hi; ++p) mx = changed(p) ? p : mx;
        int inc = mx;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFullMask, inc, o);
            if (lane >= o) inc = max(inc, t);
        }
        if (lane == 31) wmax[w] = inc;
        int run = __shfl_up_sync(kFullMask, inc, 1);
        if (lane == 0) run = 0;
        __syncthreads();
        for (int v = 0; v < w; ++v) run = max(run, wmax[v]);
        for (int p = lo; p < hi; ++p) {
            run = changed(p) ? p : run;
            last[p] = (unsigned short)run;
        }
    }
    double mean = 0.0, M2 = 0.0;
    const double* a = sA + lane * (kStatChunk + 1);  // the lane's chunk: element k at k + k / 256
    if (w == 0) {
        for (int k0 = 0; k0 < (int)m; k0 += 32) {
            const double rl = __drcp_rn((double)(k0 + lane + 1));
            const int kn = min(32, (int)m - k0);
#pragma unroll 4
            for (int k = 0; k < kn; ++k) {
                const double r = __shfl_sync(kFullMask, rl, k);
                const double x = a[k0 + k + ((k0 + k) >> 8)];
                const double delta = __dsub_rn(x, mean);
                mean = __dadd_rn(mean, quotient(delta, (double)(k0 + k + 1), r));
                M2 = __fma_rn(delta, __dsub_rn(x, mean), M2);
            }
        }
    }
    const double inv_m = 1.0 / (double)m;
    for (int t = 0; t <= kStatChunk / 32; ++t) {
        if (w == 0 && t < kStatChunk / 32) {
            double* mb = buf + (t & 1) * 2 * kStatBatch + lane * 33;
#pragma unroll 4
            for (int k = 0; k < 32; ++k) {
                const int i = t * 32 + k;
                if (i > 0) {
                    const int e = i + (int)m - 1;
                    const double xin = a[e + (e >> 8)], xout = a[i - 1];  // i - 1 < 256
                    const double d = __dsub_rn(xin, xout);
                    const double mnew = __fma_rn(d, inv_m, mean);
                    M2 = __fma_rn(d, __dsub_rn(__dadd_rn(__dsub_rn(xin, mnew), xout), mean), M2);
                    mean = mnew;
                }
                mb[k] = mean;
                mb[kStatBatch + k] = M2;
            }
        } else if (w > 0 && t > 0) {
            const double* mb = buf + ((t - 1) & 1) * 2 * kStatBatch;
            for (int e = tid - 32; e < 1024; e += kStatThreads - 32) {
                const int c = e >> 5, k = e & 31;
                const int i = c * kStatChunk + (t - 1) * 32 + k;
                if (base + i < PL) {
                    const double q = mb[kStatBatch + c * 33 + k];
                    const bool flat = last[i + (int)m - 1] <= i;
                    mean_out[base + i] = mb[c * 33 + k];
                    norm_out[base + i] = (flat || !(q > 0.0)) ? __longlong_as_double(0x7ff8000000000000ll)
                                                              : 1.0 / sqrt(q);
                }
            }
        }
        __syncthreads();
    }
}

// FP32 records.  For window i (i < PL):
//   df[i] = (A[i+m] - A[i]) / 2,  dg[i] = (A[i+m] - mean[i+1]) + (A[i] - mean[i])
// (zero for the last window, whose successor does not exist), nn[i] = norm[i].
// Row records are stored as pairs (x[j], x[j+H]) for the f32x2 datapath:
//   rowrec[j] = {df[j], df[j+H], dg[j], dg[j+H], nn[j], nn[j+H], 1, 1}
// Column records duplicate and negate the column terms:
//   colrec[p] = {-df[p], -df[p], -dg[p], -dg[p], nn[p], nn[p], 1/nn[p], 1/nn[p]}
// Entries past PL read as df = dg = 0, nn = NaN.
__device__ __forceinline__ void fp32_terms(const double* A, int64_t m, int64_t PL,
                                           const double* mean, const double* norm, int64_t i,
                                           float& df, float& dg, float& nn) {
    if (i >= PL) {
        df = 0.f;
        dg = 0.f;
        nn = __int_as_float(0x7fffffff);
        return;
    }
    if (i + 1 < PL) {
        const double xin = A[i + m], xout = A[i];
        df = (float)((xin - xout) * 0.5);
        dg = (float)((xin - mean[i + 1]) + (xout - mean[i]));
    } else {
        df = 0.f;
        dg = 0.f;
    }
    nn = (float)norm[i];
}

__device__ __forceinline__ void pack_fp32_record(const double* A, int64_t m, int64_t PL, int H,
                                                 const double* mean, const double* norm, int64_t j,
                                                 float4* rowrec, float4* colrec) {
    float df0, dg0, nn0, df1, dg1, nn1;
    fp32_terms(A, m, PL, mean, norm, j, df0, dg0, nn0);
    fp32_terms(A, m, PL, mean, norm, j + H, df1, dg1, nn1);
    rowrec[2 * j] = make_float4(df0, df1, dg0, dg1);
    rowrec[2 * j + 1] = make_float4(nn0, nn1, 1.f, 1.f);
    colrec[2 * j] = make_float4(-df0, -df0, -dg0, -dg0);
    const float inv = 1.f / nn0;
    colrec[2 * j + 1] = make_float4(nn0, nn0, inv, inv);
}

}  // namespace mpgpu
