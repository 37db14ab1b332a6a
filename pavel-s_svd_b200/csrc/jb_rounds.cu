// jb_rounds.cu - the rounds of the block Jacobi (svdbench/standalone/solvers.py:
// 30-68) on a batch of float64 matrices: one launch a round and one pair of
// launches for the convergence test.
//
// A round's pairs of column groups are orthogonalised by one CTA each: the
// columns W[:, cols] are gathered into shared memory and rotated there by
// group_sweeps (jb_group.cuh), which gives V_ij, its columns by descending norm;
// W[:, cols] <- W[:, cols] V_ij and V[:, cols] <- V[:, cols] V_ij follow in the
// same CTA, a thread a row.  W and V are kept transposed (a column contiguous),
// so gathers and write-backs are runs of a column.  The products take the old
// W, as the reference does: writing the rotated columns back costs the same and
// leaves the polar factor's error 12 % larger.  Bound by the latency of the
// Jacobi steps (7 CTAs of two warps an SM).  256 x 96 x 64, blocks of 8, a round
// of 1024 pairs of 96 x 16: 105 us; the batched solve of the pairs, two gathers,
// two GEMMs and two scatters took 285.
#include <cuda_runtime.h>
#include <stdint.h>
#include "jacobi_b200.h"
#include "jb_device.cuh"
#include "jb_group.cuh"

namespace jb {
namespace rnd {

constexpr int kMaxRows = 128, kMaxCols = 32;

struct PairParams {
    double *Wt, *Vt;          // (batch, n, m), (batch, n, n): row j = column j
    const int32_t *cols;      // (pairs, c)
    int32_t *status, *sweeps; // (batch * pairs)
    int m, n, pairs, c, max_sweeps;
    double tol;
};

template <int GL, int B, int RW, int RV, int THREADS>
__global__ void __launch_bounds__(THREADS) pair_kernel(PairParams p) {
    using C = GroupCfg<double, 1, GL, B, RW, RV>;
    constexpr int LD = C::LD, CM = (2 * B * THREADS / GL) < C::NCOLS ? (2 * B * THREADS / GL) : C::NCOLS;
    constexpr int WARPS = THREADS / 32;
    extern __shared__ __align__(16) double area[];        // np columns: W, then V_ij
    __shared__ double s_scales[kMaxCols], s_red[32], s_norm[kMaxCols];
    __shared__ int s_cols[kMaxCols], s_order[kMaxCols];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t z = blockIdx.x / p.pairs;
    const int c = p.c, m = p.m, n = p.n, np = 2 * B * ((c + 2 * B - 1) / (2 * B));
    double *W = p.Wt + z * n * m, *V = p.Vt + z * n * n;
    if (tid < c) s_cols[tid] = p.cols[(int64_t)(blockIdx.x % p.pairs) * c + tid];
    for (int i = tid; i < np * LD / 2; i += THREADS) ((double2 *)area)[i] = make_double2(0.0, 0.0);
    team_sync<THREADS>();
    // the columns, and a power of two that keeps their squares in range
    double amax = 0.0;
    int bad = 0;
    for (int j = warp; j < c; j += WARPS) {
        const double *col = W + (int64_t)s_cols[j] * m;
        for (int i = lane; i < m; i += 32) {
            const double x = col[i];
            if (!isfinite(x)) bad = 1;
            amax = fmax(amax, fabs(x));
            area[j * LD + i] = x;
        }
        if (lane == 0) area[j * LD + C::VOFF + j] = 1.0;
    }
    amax = warp_max(amax);
    if (lane == 0) s_red[warp] = amax;
    bad = THREADS == 32 ? __any_sync(FULL, bad) : __syncthreads_or(bad);
    team_sync<THREADS>();
#pragma unroll
    for (int w = 0; w < WARPS; ++w) amax = fmax(amax, s_red[w]);
    int ns = 0, st = JB_ST_NONFINITE_IN, e = 0;
    if (!bad) {
        if (amax > 0.0) frexp(amax, &e);
        if (e)
            for (int j = warp; j < c; j += WARPS)
                for (int i = lane; i < m; i += 32) area[j * LD + i] = dscale(area[j * LD + i], -e);
        team_sync<THREADS>();
        bool conv;
        ns = group_sweeps<double, 1, GL, B, RW, RV, THREADS>(area, c, p.tol, p.max_sweeps, s_scales, s_red, conv);
        st = conv ? JB_ST_OK : JB_ST_NOT_CONVERGED;
    }
    if (st == JB_ST_OK) {
        for (int j = warp; j < c; j += WARPS) {
            double s = 0.0;
            for (int i = lane; i < m; i += 32) s = dfma(area[j * LD + i], area[j * LD + i], s);
            s = warp_sum(s);
            if (lane == 0) s_norm[j] = s;
        }
        team_sync<THREADS>();
        if (tid < c) {                                     // descending, the first of equals first
            int r = 0;
            for (int j = 0; j < c; ++j) r += s_norm[j] > s_norm[tid] || (s_norm[j] == s_norm[tid] && j < tid);
            s_order[r] = tid;
        }
        team_sync<THREADS>();
        for (int r = tid; r < m + n; r += THREADS) {       // a row of W or V: read whole, then written
            double *at = r < m ? W + r : V + (r - m);
            const int64_t ld = r < m ? m : n;
            double x[CM];
#pragma unroll
            for (int j = 0; j < CM; ++j) x[j] = j < c ? at[s_cols[j] * ld] : 0.0;
            for (int k = 0; k < c; ++k) {
                const double2 *v = (const double2 *)(area + s_order[k] * LD + C::VOFF);
                double a = 0.0, b = 0.0;
#pragma unroll
                for (int j = 0; j < CM / 2; ++j) {
                    const double2 y = v[j];
                    a = dfma(x[2 * j], y.x, a);
                    b = dfma(x[2 * j + 1], y.y, b);
                }
                at[s_cols[k] * ld] = a + b;
            }
        }
    }
    if (tid == 0) {
        p.status[blockIdx.x] = st;
        p.sweeps[blockIdx.x] = ns;
    }
}

template <int GL, int B, int RW, int RV, int THREADS>
static int launch_pairs(const PairParams &p, int64_t grid, cudaStream_t st) {
    using C = GroupCfg<double, 1, GL, B, RW, RV>;
    const size_t smem = (size_t)(2 * B * ((p.c + 2 * B - 1) / (2 * B))) * C::LD * 8;
    auto kern = pair_kernel<GL, B, RW, RV, THREADS>;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    kern<<<(unsigned)grid, THREADS, smem, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

// d[z, j] = ||column j||^2; one warp a column.
__global__ void __launch_bounds__(256) norms2_kernel(const double *Wt, double *d, int64_t columns, int m,
                                                     unsigned long long *worst) {
    const int64_t j = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) *worst = 0ull;
    if (j >= columns) return;
    double s = 0.0;
    for (int i = lane; i < m; i += 32) s = dfma(Wt[j * m + i], Wt[j * m + i], s);
    s = warp_sum(s);
    if (lane == 0) d[j] = s;
}

// The largest |g_pq| / sqrt(g_pp g_qq) over pairs of live columns (d_j > floor
// max d) of every matrix, as the bits of a double (NaN above all).  A CTA has
// one 32 x 32 tile p >= q of one matrix, a warp a 16 x 16 part of it on the
// FP64 matrix unit, its operands straight from L2 (every column is read by
// n / 32 CTAs).
__global__ void __launch_bounds__(128) worst_kernel(const double *Wt, const double *d, int m, int n, int tiles,
                                                    double floor2, unsigned long long *worst) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t z = blockIdx.x / tiles;
    const int tt = blockIdx.x % tiles;
    int ti = (int)((sqrtf(8.f * (float)tt + 1.f) - 1.f) * 0.5f);
    while (ti * (ti + 1) / 2 > tt) --ti;
    while ((ti + 1) * (ti + 2) / 2 <= tt) ++ti;
    const int p0 = 32 * ti + 16 * (warp >> 1), q0 = 32 * (tt - ti * (ti + 1) / 2) + 16 * (warp & 1);
    const double *W = Wt + z * n * m, *dz = d + z * n;
    double dmax = 0.0;
    for (int j = lane; j < n; j += 32) dmax = dz[j] > dmax ? dz[j] : dmax;
    dmax = warp_max(dmax);
    double acc[2][2][2] = {};
    if (p0 < n && q0 < n) {
        const double *pa[2], *pb[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {                      // columns past the last: the last, not used
            const int jp = p0 + 8 * r + (lane >> 2), jq = q0 + 8 * r + (lane >> 2);
            pa[r] = W + (int64_t)(jp < n ? jp : n - 1) * m;
            pb[r] = W + (int64_t)(jq < n ? jq : n - 1) * m;
        }
#pragma unroll 4
        for (int k0 = 0; k0 < m; k0 += 4) {
            const int k = k0 + (lane & 3);
            double x[2], y[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                x[r] = k < m ? pa[r][k] : 0.0;
                y[r] = k < m ? pb[r][k] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                 : "+d"(acc[r][s][0]), "+d"(acc[r][s][1])
                                 : "d"(x[r]), "d"(y[s]));
        }
    }
    unsigned long long best = 0ull;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int jp = p0 + 8 * r + (lane >> 2), jq = q0 + 8 * s + 2 * (lane & 3) + e;
                if (jp < n && jq < n && jp != jq) {
                    const double a = dz[jp], b = dz[jq];
                    if (!(a <= floor2 * dmax) && !(b <= floor2 * dmax)) {
                        const double den = sqrt(a) * sqrt(b);
                        const unsigned long long x = (unsigned long long)__double_as_longlong(
                            fabs(acc[r][s][e]) / (den < 2.2250738585072014e-308 ? 2.2250738585072014e-308 : den));
                        best = x > best ? x : best;
                    }
                }
            }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(FULL, best, o);
        best = x > best ? x : best;
    }
    if (lane == 0 && best) atomicMax(worst, best);
}

}  // namespace rnd
}  // namespace jb

using namespace jb::rnd;

extern "C" {

// Lanes a block pair and rows a lane from the shape, as the batched float64
// solve's (launch_group, jb_batched.cu), with forms for 8 columns (one warp)
// and for 96 rows: a lane's registers hold no more padding than a third.
int jb_pair_round_f64(double *Wt, double *Vt, const int32_t *cols, int64_t batch, int32_t m, int32_t n, int32_t pairs,
                      int32_t c, double tol, int32_t max_sweeps, int32_t *status, int32_t *sweeps, void *stream) {
    if (!Wt || !Vt || !cols || !status || !sweeps || batch < 0 || n < 2 || m < n || pairs < 0 || c < 2 || c > n ||
        max_sweeps < 1)
        return JB_EINVAL;
    if (m > kMaxRows || c > kMaxCols || batch * pairs > 0x7fffffff) return JB_ETOOBIG;
    if (batch == 0 || pairs == 0) return JB_OK;
    PairParams p{Wt, Vt, cols, status, sweeps, m, n, pairs, c, max_sweeps,
                 tol > 0 ? tol : 10 * 2.220446049250313e-16};
    const int64_t grid = batch * pairs;
    cudaStream_t st = (cudaStream_t)stream;
    if (c <= 8) {
        if (m <= 64) return launch_pairs<16, 2, 4, 2, 32>(p, grid, st);
        if (m <= 96) return launch_pairs<16, 2, 6, 2, 32>(p, grid, st);
        return launch_pairs<16, 2, 8, 2, 32>(p, grid, st);
    }
    if (c <= 16) {
        if (m <= 32) return launch_pairs<8, 2, 4, 2, 32>(p, grid, st);
        if (m <= 64) return launch_pairs<16, 2, 4, 2, 64>(p, grid, st);
        if (m <= 96) return launch_pairs<16, 2, 6, 2, 64>(p, grid, st);
        return launch_pairs<16, 2, 8, 2, 64>(p, grid, st);
    }
    if (m <= 64) return launch_pairs<8, 2, 8, 4, 64>(p, grid, st);
    if (m <= 96) return launch_pairs<16, 2, 6, 2, 128>(p, grid, st);
    return launch_pairs<16, 2, 8, 2, 128>(p, grid, st);
}

int jb_worst_correlation_f64(const double *Wt, int64_t batch, int32_t m, int32_t n, double live, double *norms2,
                             double *worst, void *stream) {
    if (!Wt || !norms2 || !worst || batch < 1 || m < 1 || n < 1) return JB_EINVAL;
    const int nt = (n + 31) / 32;
    const int64_t columns = batch * n, tiles = (int64_t)nt * (nt + 1) / 2;
    if (n > 32768 || (columns + 7) / 8 > 0x7fffffff || batch * tiles > 0x7fffffff) return JB_ETOOBIG;
    cudaStream_t st = (cudaStream_t)stream;
    norms2_kernel<<<(unsigned)((columns + 7) / 8), 256, 0, st>>>(Wt, norms2, columns, m, (unsigned long long *)worst);
    if (cudaGetLastError() != cudaSuccess) return JB_ECUDA;
    worst_kernel<<<(unsigned)(batch * tiles), 128, 0, st>>>(Wt, norms2, m, n, (int)tiles, live * live,
                                                           (unsigned long long *)worst);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

}  // extern "C"
