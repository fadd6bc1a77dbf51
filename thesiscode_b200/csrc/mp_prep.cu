// Per-window preparation kernels: window statistics, first dot products and
// the packed row/column records the join kernels stream.
//
// Two statistics paths:
//  * reference-exact (FP64 form): the reference's prefix-sum formula,
//    scrimppp/src/ScrimpSequOpt.cpp:33-79, evaluated with explicitly rounded
//    operations (__dadd_rn/__dmul_rn/... are never contracted into FMAs) so the
//    result is bit-identical to the reference built with IEEE semantics.  The
//    two prefix sums are dependent chains, each on a lane of its own (prefix_block).
//  * FP64 Welford (FP32 form): Welford's mean/M2 update slides over chunks of
//    256 windows, restarting from a fresh Welford pass at every chunk start;
//    exact zero-variance windows are found from the places where the value
//    changes, so a constant window at any level is flagged exactly.
#include <atomic>

#include "mp_common.cuh"
#include "mp_kernels.h"
#include "mp_prep_device.cuh"

namespace mpgpu {

// ---- reference-exact statistics -------------------------------------------

__global__ void __launch_bounds__(kPrefixThreads)
    ref_prefix_kernel(const double* __restrict__ A, int64_t n, double* __restrict__ cs,
                      double* __restrict__ cs2) {
    __shared__ __align__(16) char buf[PrefixSmem<kPrefixChunk>::kBytes];
    if (blockIdx.x == 0) prefix_block<kPrefixChunk>(A, n, cs, cs2, buf);
}

// Window sums from prefix differences, mean = S/m, var = S2/m - mean^2,
// sInv = 1/sqrt(var), muS = (mean*sInv)*sqrt(m) (ScrimpSequOpt.cpp:50-68).
__global__ void ref_stats_kernel(const double* __restrict__ cs, const double* __restrict__ cs2,
                                 int64_t PL, int64_t m, double* __restrict__ muS,
                                 double* __restrict__ sInv) {
    const double dm = (double)m;
    const double sqrt_m = __dsqrt_rn(dm);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < PL;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double s = (i == 0) ? cs[m - 1] : __dsub_rn(cs[m - 1 + i], cs[i - 1]);
        const double s2 = (i == 0) ? cs2[m - 1] : __dsub_rn(cs2[m - 1 + i], cs2[i - 1]);
        const double mean = __ddiv_rn(s, dm);
        const double var = __dsub_rn(__ddiv_rn(s2, dm), __dmul_rn(mean, mean));
        const double si = __ddiv_rn(1.0, __dsqrt_rn(var));
        sInv[i] = si;
        muS[i] = __dmul_rn(__dmul_rn(mean, si), sqrt_m);
    }
}

// First dot product per diagonal, summed in k order without fusion
// (ScrimpSequOpt.cpp:81-96).  Consecutive threads take consecutive diagonals
// so the A[k+d] reads coalesce and A[k] is a broadcast.
__global__ void first_qt_kernel(const double* __restrict__ A, int64_t m, int64_t d_lo,
                                int64_t d_hi, double* __restrict__ qt) {
    for (int64_t d = d_lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; d < d_hi;
         d += (int64_t)gridDim.x * blockDim.x) {
        double z = 0.0;
        const double* a = A + d;
        for (int64_t k = 0; k < m; ++k) z = __dadd_rn(z, __dmul_rn(__ldg(a + k), __ldg(A + k)));
        qt[d - d_lo] = z;
    }
}

// Row/column record of the FP64 join: {A[i], A[i+m], sInv[i], muS[i]}; sInv[i], no
// longer needed, becomes Fp64BandParams::colgate.
// `Apad` holds n+1 values (A[n] = 0 feeds only the update after a diagonal's
// last cell, whose result is never used).
__global__ void pack_fp64_kernel(const double* __restrict__ Apad, int64_t m, int64_t count,
                                 double* __restrict__ sInv, const double* __restrict__ muS,
                                 double4* __restrict__ rec) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double s = sInv[i];
        sInv[i] = fp64_gate_mean(s, muS[i]);
        rec[i] = make_double4(Apad[i], Apad[i + m], s, muS[i]);
    }
}

// ---- FP64 Welford statistics (FP32 form) ----------------------------------

// chg[i] = 1 if A[i] != A[i-1] (i >= 1), chg[0] = 0; an inclusive scan of chg
// gives the number of value changes up to i.
__global__ void change_flags_kernel(const double* __restrict__ A, int64_t n, int* __restrict__ chg) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        chg[i] = (i > 0 && A[i] != A[i - 1]) ? 1 : 0;
}

// Block-level inclusive scan helper (Hillis-Steele over a warp, then warps).
__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFullMask, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Two-level inclusive scan of int flags: per-block scan + block totals.
__global__ void scan_blocks_kernel(int* __restrict__ x, int64_t n, int* __restrict__ block_tot) {
    __shared__ int wsum[32];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int v = (i < n) ? x[i] : 0;
    v = warp_incl_scan(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 31) wsum[w] = v;
    __syncthreads();
    if (w == 0) {
        int t = (lane < (int)(blockDim.x >> 5)) ? wsum[lane] : 0;
        t = warp_incl_scan(t);
        wsum[lane] = t;
    }
    __syncthreads();
    if (w > 0) v += wsum[w - 1];
    if (i < n) x[i] = v;
    if (threadIdx.x == blockDim.x - 1) block_tot[blockIdx.x] = v;
}

__global__ void scan_totals_kernel(int* __restrict__ tot, int64_t nblocks) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int s = 0;
    for (int64_t b = 0; b < nblocks; ++b) {
        s += tot[b];
        tot[b] = s;
    }
}

__global__ void scan_add_kernel(int* __restrict__ x, int64_t n, const int* __restrict__ tot) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n && blockIdx.x > 0) x[i] += tot[blockIdx.x - 1];
}

// Welford statistics per chunk of windows (see welford_chunk).
__global__ void welford_kernel(const double* __restrict__ A, int64_t m, int64_t PL, int64_t chunk,
                               const int* __restrict__ nchg, double* __restrict__ mean_out,
                               double* __restrict__ norm_out) {
    const int64_t nthreads = (PL + chunk - 1) / chunk;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nthreads;
         t += (int64_t)gridDim.x * blockDim.x)
        welford_chunk(A, m, PL, chunk, t, nchg, mean_out, norm_out);
}

// Welford statistics, one block per 32 chunks (see stat_block); the zeros behind the
// series and the statistics, too (their places are read by nothing here).
__global__ void __launch_bounds__(kStatThreads)
    stat_kernel(double* A, int64_t m, int64_t PL, int64_t pad, double* mean, double* norm) {
    extern __shared__ __align__(16) char smem_stat[];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < pad;
         i += (int64_t)gridDim.x * blockDim.x) {
        A[PL + m - 1 + i] = 0.0;
        mean[PL + i] = 0.0;
        norm[PL + i] = 0.0;
    }
    stat_block(A, m, PL, (int64_t)blockIdx.x * kStatSpan, mean, norm, smem_stat);
}

void configure_stats() {
    cudaFuncSetAttribute(stat_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)stat_smem_bytes(kStatMaxM));
}

int launch_fp32_stats(double* A, int64_t m, int64_t PL, int64_t pad, int* nchg, int* tot, double* mean,
                      double* norm, cudaStream_t s) {
    const int64_t n = PL + m - 1;
    if (m <= kStatMaxM) {
        // per-device attribute, idempotent: see launch_fp32_join
        static std::atomic<unsigned long long> configured{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            configure_stats();
            configured.fetch_or(bit, std::memory_order_release);
        }
        stat_kernel<<<(unsigned)((PL + kStatSpan - 1) / kStatSpan), kStatThreads, stat_smem_bytes(m), s>>>(
            A, m, PL, pad, mean, norm);
        return 1;
    }
    constexpr int T = 256;
    const int64_t nblk = (n + T - 1) / T;
    cudaMemsetAsync(A + n, 0, 8 * pad, s);
    cudaMemsetAsync(mean + PL, 0, 8 * pad, s);
    cudaMemsetAsync(norm + PL, 0, 8 * pad, s);
    change_flags_kernel<<<grid_for(n), T, 0, s>>>(A, n, nchg);
    scan_blocks_kernel<<<(unsigned)nblk, T, 0, s>>>(nchg, n, tot);
    scan_totals_kernel<<<1, 1, 0, s>>>(tot, nblk);
    scan_add_kernel<<<(unsigned)nblk, T, 0, s>>>(nchg, n, tot);
    welford_kernel<<<grid_for((PL + kStatChunk - 1) / kStatChunk), T, 0, s>>>(A, m, PL, kStatChunk, nchg, mean,
                                                                              norm);
    return 5;
}

// Row and column records of the FP32 form (see pack_fp32_record), the keys and,
// for a launch over one descriptor, that descriptor and the tile counter.
__global__ void pack_fp32_kernel(const double* __restrict__ A, int64_t m, int64_t PL, int H,
                                 int64_t count, const double* __restrict__ mean,
                                 const double* __restrict__ norm, float4* __restrict__ rowrec,
                                 float4* __restrict__ colrec, unsigned long long* __restrict__ key,
                                 unsigned long long init, const Fp32TileParams P,
                                 Fp32TileParams* __restrict__ desc, unsigned long long* __restrict__ counter) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < count;
         j += (int64_t)gridDim.x * blockDim.x) {
        pack_fp32_record(A, m, PL, H, mean, norm, j, rowrec, colrec);
        if (j < PL) key[j] = fp32_first_key(init, norm[j]);
        if (j == 0 && desc) *desc = P;
        if (j == 0 && counter) *counter = 0;
    }
}

}  // namespace mpgpu
