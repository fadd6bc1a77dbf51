// PreSCRIMP: the anytime front end of SCRIMP++ (scrimppp/src/ScrimpppOrig.cpp:130-266).
//
// Query windows i = 0, s, 2s, ... (s = floor(stride * m)) each get their whole
// distance profile; every cell updates both windows' profile entries; then,
// from each query's best neighbour j, the diagonal j - i is walked s - 1 cells
// forward and backward with the reference's running dot product.  The
// reference computes the query rows by FFT convolution (FFTW); here each cell
// is a direct FP64 dot product over the window, tiled so that a CTA serves 32
// queries x 256 windows from shared memory (m DFMA per cell, no FFT, and more
// accurate than the FFT's rounding).  All updates are min-merges of 64-bit
// keys, so the result does not depend on the (shuffled, in the reference)
// query order.
#include <cfloat>
#include <type_traits>

#include "mp_common.cuh"
#include "mp_kernels.h"

namespace mpgpu {

namespace {

constexpr int kQB = 32;          // queries per CTA, all of them in every warp
constexpr int kJW = 64;          // windows per warp
constexpr int kRowWarps = 4;     // warps per CTA
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kJB = kRowWarps * kJW;  // windows per CTA; a query's best of them is one merge
constexpr int kKC = 32;          // window elements per shared-memory stage
constexpr int kQS = kKC + 4;     // doubles between a stage's queries: conflict-free A fragments
constexpr int kWN = kJB + kKC;   // series values per stage
constexpr int kStage = kQB * kQS + kWN;  // doubles per stage
constexpr unsigned long long kNone = ~0ull;

// Distance keys: ord(d) min-merged (exact); index keys: ord(d) with its low
// idx_bits replaced by the neighbour, min-merged (smallest neighbour among
// distances equal to ~2^-(52-idx_bits+12) relative).
__device__ __forceinline__ void merge(unsigned long long* kex, unsigned long long* kix, int64_t w,
                                      double d, int64_t nb, int idx_bits) {
    const unsigned long long o = ord_f64(d);
    const unsigned long long low = (1ull << idx_bits) - 1ull;
    atomicMin(kex + w, o);
    atomicMin(kix + w, (o & ~low) | (unsigned long long)nb);
}

// The reference's distance of one cell (ScrimpppOrig.cpp:195, 226, 246):
// 2 * (m - (qt - m * mean_j * mean_i) / (sigma_j * sigma_i)), same operation order.
__device__ __forceinline__ double orig_distance(double mm, double qt, double mean_j, double mean_i,
                                                double sig_j, double sig_i) {
    const double corr = __dmul_rn(__dmul_rn(mm, mean_j), mean_i);
    const double x = __ddiv_rn(__dsub_rn(qt, corr), __dmul_rn(sig_j, sig_i));
    return __dmul_rn(2.0, __dsub_rn(mm, x));
}

}  // namespace

// ScrimpppOrig.cpp:86-107: window sums as prefix-sum differences, mean,
// variance S2/m - mean^2 and sigma = sqrt(variance).
__global__ void orig_stats_kernel(const double* __restrict__ cs, const double* __restrict__ cs2,
                                  int64_t PL, int64_t m, double* __restrict__ mean,
                                  double* __restrict__ sigma) {
    const double mm = (double)m;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < PL;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double s = i == 0 ? cs[m - 1] : __dsub_rn(cs[m - 1 + i], cs[i - 1]);
        const double s2 = i == 0 ? cs2[m - 1] : __dsub_rn(cs2[m - 1 + i], cs2[i - 1]);
        const double mu = __ddiv_rn(s, mm);
        mean[i] = mu;
        sigma[i] = __dsqrt_rn(__dsub_rn(__ddiv_rn(s2, mm), __dmul_rn(mu, mu)));
    }
}

__global__ void prescrimp_keys_init_kernel(unsigned long long* __restrict__ a, int64_t count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
         i += (int64_t)gridDim.x * blockDim.x)
        a[i] = kNone;
}

// Query rows: CTA b covers windows [wt*256, wt*256+256) and queries
// [qt*32, qt*32+32), wt = b % window tiles, qt = b / window tiles (a 1-D grid,
// so any number of queries fits).  The dot products are a matrix product,
// queries x elements by elements x windows, on the FP64 matrix instruction: a warp
// takes 32 queries x 64 windows (4 x 8 blocks), each cell accumulated in k order;
// both operands come straight from stages of the series in shared memory (window w's
// element k is value w + k), 12 reads per 32 instructions.  The next stage is copied
// in while one runs.
// What bounds it: the FP64 pipe, m operations per cell, and the distances, as many
// instructions per cell as m = 256 matrix ones; three CTAs per SM overlap the two.
// 200,003 samples, m = 256, stride 0.25 (1.6e11 operations, 8.8 ms at the pipe's
// rate): 11.5 ms (12.6 with two CTAs, 13.6 with one of 8 warps).  8 queries x 4
// windows per thread in multiply-adds took 16.0, 8 x 8 with the windows sliding
// through registers 16.9.
__global__ void __launch_bounds__(kRowThreads, 3) prescrimp_rows_kernel(const PreScrimpParams P) {
    extern __shared__ __align__(16) double smem_rows[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int lr = lane >> 2, lc = lane & 3;  // fragment row and column
    const int64_t nwt = (P.PL + kJB - 1) / kJB;
    const int64_t j0 = ((int64_t)blockIdx.x % nwt) * kJB;
    const int64_t t0 = ((int64_t)blockIdx.x / nwt) * kQB;
    // a thread copies element threadIdx.x % 32 of queries threadIdx.x / 32 + 4 i, and
    // series values threadIdx.x + 128 i
    const int qk = threadIdx.x & 31, q0 = threadIdx.x >> 5;
    const double* qsrc = P.A + (t0 + q0) * P.step + qk;
    const int nq = (int)min((int64_t)kQB, P.Q - t0);  // queries of the tile
    auto load = [&](int64_t k0, int buf) {
        double* sq = smem_rows + buf * kStage;
        double* sw = sq + kQB * kQS;
#pragma unroll
        for (int i = 0; i < kQB / kRowWarps; ++i) {
            const int q = q0 + kRowWarps * i;
            const bool in = q < nq && k0 + qk < P.m;
            cp_async8_or_zero(sq + q * kQS + qk, in ? qsrc + kRowWarps * i * P.step + k0 : P.A, in);
        }
        const int64_t left = P.n - j0 - k0;  // zero past the series: only cells j >= PL read it
        for (int e = threadIdx.x; e < kWN; e += kRowThreads)
            cp_async8_or_zero(sw + e, e < left ? P.A + j0 + k0 + e : P.A, e < left);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double acc[4][8][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
    load(0, 0);
    int buf = 0;
    for (int64_t k0 = 0; k0 < P.m; k0 += kKC, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (k0 + kKC < P.m) load(k0 + kKC, buf ^ 1);
        const double* sq = smem_rows + buf * kStage + lr * kQS + lc;
        const double* sw = smem_rows + buf * kStage + kQB * kQS + wi * kJW + lr + lc;
        const int kn = (int)min((int64_t)kKC, P.m - k0);
        auto step = [&](int kk, bool in) {  // elements kk .. kk + 3; in: the lane's is one of the m
            double a[4], b[8];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = in ? sq[8 * r * kQS + kk] : 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c) b[c] = in ? sw[8 * c + kk] : 0.0;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) mma_f64(acc[r][c], a[r], b[c]);
        };
        int kk = 0;
#pragma unroll 2
        for (; kk + 4 <= kn; kk += 4) step(kk, true);
        if (kk < kn) step(kk, kk + lc < kn);  // 0 * 0 for the elements past m
    }
    // distances; per query the warp's best window, per window its best query
    const double mm = (double)P.m;
    double rb[4];
    int ri[4];
    double mi[4], si[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t t = t0 + 8 * r + lr;
        rb[r] = DBL_MAX;
        ri[r] = -1;
        mi[r] = t < P.Q ? P.mean[t * P.step] : 0.0;
        si[r] = t < P.Q ? P.sigma[t * P.step] : 0.0;
    }
    // positions as unsigned numbers: a tile may reach beyond 2^31 - 1
    const unsigned i0 = (unsigned)(t0 * P.step), jw = (unsigned)j0 + wi * kJW, PL = (unsigned)P.PL;
    const unsigned step = (unsigned)min(P.step, P.PL), excl = (unsigned)min(P.excl, P.PL);
    // A product of deviations that is 0 (a constant window) or NaN: the division's steps
    // for such operands cost several times its ordinary ones, and a test per cell costs the
    // ordinary ones 3%, so only a warp that has such a window tests (100,000 samples, m =
    // 64, all constant: 9.6 ms a call without the test, 5.1 with it; a walk 5.5).
    constexpr double kInf = __builtin_huge_val();
    auto distances = [&](auto degenerate) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned j = jw + 8 * c + 2 * lc + h;
                double cb = DBL_MAX;
                int ci = -1;
                if (j < PL) {
                    const double mj = __dmul_rn(mm, P.mean[j]), sj = P.sigma[j];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int q = 8 * r + lr;
                        const unsigned i = i0 + q * step;
                        if (q >= nq || prescrimp_excluded(i, j, excl)) continue;
                        // orig_distance
                        const double x = __dsub_rn(acc[r][c][h], __dmul_rn(mj, mi[r])), y = __dmul_rn(sj, si[r]);
                        double z;
                        if (decltype(degenerate)::value && !(y > 0.0))
                            z = __dmul_rn(x, y == 0.0 ? copysign(kInf, y) : y);
                        else
                            z = __ddiv_rn(x, y);
                        const double d = __dmul_rn(2.0, __dsub_rn(mm, z));
                        if (d < cb) {
                            cb = d;
                            ci = (int)i;
                        }
                        if (d < rb[r]) {
                            rb[r] = d;
                            ri[r] = (int)j;
                        }
                    }
                }
                // over the warp's queries, the smallest among equals
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const double d = __shfl_xor_sync(kFullMask, cb, o);
                    const int i = __shfl_xor_sync(kFullMask, ci, o);
                    if (i >= 0 && (ci < 0 || d < cb || (d == cb && i < ci))) {
                        cb = d;
                        ci = i;
                    }
                }
                if (lr == 0 && ci >= 0) merge(P.kex, P.kix, j, cb, ci, P.idx_bits);
            }
        }
    };
    bool odd = false;
#pragma unroll
    for (int r = 0; r < 4; ++r) odd |= t0 + 8 * r + lr < P.Q && !(si[r] > 0.0);
#pragma unroll
    for (int e = 0; e < kJW; e += 32) odd |= jw + e + lane < PL && !(P.sigma[jw + e + lane] > 0.0);
    if (__any_sync(kFullMask, odd))
        distances(std::true_type{});
    else
        distances(std::false_type{});
    __syncthreads();  // the stages are free
    double* rbest = smem_rows;                                   // [kRowWarps][kQB]
    int* ridx = reinterpret_cast<int*>(rbest + kRowWarps * kQB);  // [kRowWarps][kQB]
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const double d = __shfl_xor_sync(kFullMask, rb[r], o);
            const int j = __shfl_xor_sync(kFullMask, ri[r], o);
            if (j >= 0 && (ri[r] < 0 || d < rb[r] || (d == rb[r] && j < ri[r]))) {
                rb[r] = d;
                ri[r] = j;
            }
        }
        if (lc == 0) {
            rbest[wi * kQB + 8 * r + lr] = rb[r];
            ridx[wi * kQB + 8 * r + lr] = ri[r];
        }
    }
    __syncthreads();
    if (threadIdx.x < kQB) {
        const int q = threadIdx.x;
        double b = DBL_MAX;
        int bj = -1;
        for (int v = 0; v < kRowWarps; ++v) {
            const int j = ridx[v * kQB + q];
            if (j >= 0 && (bj < 0 || rbest[v * kQB + q] < b)) {
                b = rbest[v * kQB + q];
                bj = j;
            }
        }
        if (bj >= 0) {
            merge(P.rex, P.rix, t0 + q, b, bj, P.idx_bits);                // the row's own best
            merge(P.kex, P.kix, (t0 + q) * P.step, b, bj, P.idx_bits);     // profile[i]
        }
    }
}

// Diagonal walks from each query's best neighbour (ScrimpppOrig.cpp:212-255):
// thread 2t walks forward, 2t+1 backward, s - 1 cells each.
__global__ void prescrimp_refine_kernel(const PreScrimpParams P) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t t = g >> 1;
    if (t >= P.Q) return;
    const bool fwd = (g & 1) == 0;
    const unsigned long long rx = P.rex[t];
    if (rx == kNone) return;
    const unsigned long long low = (1ull << P.idx_bits) - 1ull;
    const int64_t i = t * P.step;
    const int64_t j = (int64_t)(P.rix[t] & low);
    const double dmin = unord_f64(rx);
    const double mm = (double)P.m;
    const double* A = P.A;
    // lastz = (m - profile[i] / 2) * (sigma_j * sigma_i) + m * mean_j * mean_i
    double z = __dadd_rn(__dmul_rn(__dsub_rn(mm, __ddiv_rn(dmin, 2.0)),
                                   __dmul_rn(P.sigma[j], P.sigma[i])),
                         __dmul_rn(__dmul_rn(mm, P.mean[j]), P.mean[i]));
    if (fwd) {
        for (int64_t k = 1; k < P.step && i + k < P.PL && j + k < P.PL; ++k) {
            z = __dadd_rn(__dsub_rn(z, __dmul_rn(A[i + k - 1], A[j + k - 1])),
                          __dmul_rn(A[i + k + P.m - 1], A[j + k + P.m - 1]));
            const double d = orig_distance(mm, z, P.mean[j + k], P.mean[i + k], P.sigma[j + k],
                                           P.sigma[i + k]);
            if (d < DBL_MAX) {  // NaN and +inf never lower an entry (the reference's '<')
                merge(P.kex, P.kix, i + k, d, j + k, P.idx_bits);
                merge(P.kex, P.kix, j + k, d, i + k, P.idx_bits);
            }
        }
    } else {
        for (int64_t k = 1; k < P.step && i - k >= 0 && j - k >= 0; ++k) {
            z = __dadd_rn(__dsub_rn(z, __dmul_rn(A[i - k + P.m], A[j - k + P.m])),
                          __dmul_rn(A[i - k], A[j - k]));
            const double d = orig_distance(mm, z, P.mean[j - k], P.mean[i - k], P.sigma[j - k],
                                           P.sigma[i - k]);
            if (d < DBL_MAX) {
                merge(P.kex, P.kix, i - k, d, j - k, P.idx_bits);
                merge(P.kex, P.kix, j - k, d, i - k, P.idx_bits);
            }
        }
    }
}

// Keys -> squared distances (the reference's "distance") and indices; windows
// no cell reached keep the reference's initial values (+inf, 0).
__global__ void prescrimp_finalize_kernel(const unsigned long long* __restrict__ kex,
                                          const unsigned long long* __restrict__ kix, int64_t PL,
                                          int idx_bits, double* __restrict__ d2,
                                          int64_t* __restrict__ idx) {
    const unsigned long long low = (1ull << idx_bits) - 1ull;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < PL;
         i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long e = kex[i];
        if (e == kNone) {
            d2[i] = __longlong_as_double(0x7ff0000000000000ll);
            idx[i] = 0;
        } else {
            d2[i] = unord_f64(e);
            idx[i] = (int64_t)(kix[i] & low);
        }
    }
}

void launch_prescrimp(const PreScrimpParams& P, cudaStream_t s) {
    const int64_t tiles = ((P.PL + kJB - 1) / kJB) * ((P.Q + kQB - 1) / kQB);
    constexpr int smem = 2 * kStage * (int)sizeof(double);
    static_assert(smem <= 48 * 1024, "two stages within the default shared memory");
    prescrimp_rows_kernel<<<(unsigned)tiles, kRowThreads, smem, s>>>(P);
    const int64_t threads = 2 * P.Q;
    prescrimp_refine_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, s>>>(P);
}

}  // namespace mpgpu
