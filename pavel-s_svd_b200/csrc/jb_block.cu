// jb_block.cu - the non-GEMM kernels of the blocked one-sided Jacobi SVD
// (svdbench/standalone/solvers.py:30-68, block_jacobi).
//
// Block pairs live in "slots": slot k of a round holds the 2b columns of its
// pair (block i, then block j, i < j) as 2b rows of length L (columns of W
// are rows of W^T), in hi/lo BF16 parts that feed the tensor-core products.
//   jb_block_eig_f64   FP64 eigen-solve of every slot's Gram (2b x 2b):
//                      the rotation vv of the reference's inner Jacobi
//                      (solvers.py:48), written as vv^T in hi/lo BF16.
//   jb_rows_scatter    FP32 rows -> hi/lo BF16 rows at mapped positions
//                      (moves rotated blocks into the next round's slots).
//   jb_rows_combine    hi + lo BF16 rows -> FP32 rows at mapped positions.
//   jb_block_finish    sigma = column norms (FP64), descending order, cut,
//                      U = W / sigma, Vh (solvers.py:61-66 with
//                      _finish_columns :18-21).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include "jacobi_b200.h"
#include "jb_group.cuh"

namespace jb {
namespace blk {

__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ int circ(int pos, int r, int n) {
    if (pos == 0) return 0;
    int x = (pos - 1 - r) % (n - 1);
    if (x < 0) x += n - 1;
    return 1 + x;
}

constexpr int kEigThreads = 512;

// Shared-memory bytes of eig_kernel for a 2b = n slot.
__host__ __device__ inline size_t eig_smem_bytes(int n) {
    return (size_t)n * n * 8            // G, FP64
           + (size_t)n * n * 4          // Q, FP32
           + (size_t)2 * n * 8          // c/s of two rounds
           + (size_t)n * 4              // permutation
           + (size_t)(n - 1) * n        // round-robin table
           + (size_t)2 * n              // pairs of two rounds
           + 16;
}

// Q columns u, v <- [u, v] J for the column pairs b = b0, b0 + bstep, ...
__device__ __forceinline__ void rotate_q(float *Q, const unsigned char *pq, const double *cs, int n, int half, int b0,
                                         int bstep, int lane) {
    for (int b = b0; b < half; b += bstep) {
        const int u = pq[b], v = pq[half + b];
        const float fc = (float)cs[b], fs = (float)cs[half + b];
        float *qu = Q + u * n, *qv = Q + v * n;
        for (int i = lane; i < n; i += 32) {
            const float xu = qu[i], xv = qv[i];
            qu[i] = fc * xu - fs * xv;
            qv[i] = fs * xu + fc * xv;
        }
    }
}

// One CTA per slot.  G (n x n, FP64, symmetric, column-major) is rotated as
// G <- J^T G J with the one-sided Jacobi rotation of columns p, q of the slot
// (app = g_pp, aqq = g_qq, apq = g_pq; primitives.py:334-347), the pairs of a
// round in parallel (round-robin order, primitives.py:309-313), Q <- Q J
// accumulated (FP32), until no pair is active or `sweeps` sweeps.  The off
// value of the slot is the largest |g_pq| / sqrt(g_pp g_qq) over its active
// pairs of live columns (g_pp and g_qq above live_floor) in the first sweep;
// dmax is the slot's largest g_pp.
//
// Per round r: warp 0 computes the rotations of round r while the other
// warps apply round r - 1's rotations to Q (c/s and pairs double-buffered);
// one barrier; all warps rotate G with round r; one barrier.  The angle
// t = tan(theta) is formed in FP32 from exponent-scaled FP64 inputs (an
// angle error of ~1e-7 leaves |g_pq| 1e-7 of itself, which the next sweep
// removes); c = 1 / sqrt(1 + t^2) and s = t c are FP64, so every applied J
// is orthogonal to FP64 accuracy.
__global__ void __launch_bounds__(kEigThreads) eig_kernel(const float *Gin, __nv_bfloat16 *Qt_hi,
                                                          __nv_bfloat16 *Qt_lo, __nv_bfloat16 *Qt_lo2,
                                                          float *off_out, float *dmax_out, int *sweeps_out, int n,
                                                          int max_sweeps, double tol, const double *live_floor_ptr) {
    extern __shared__ __align__(16) unsigned char smem[];
    double *G = (double *)smem;                         // n x n, G[col * n + row]
    float *Q = (float *)(G + (size_t)n * n);             // n x n, Q[col * n + row]
    double *csb = (double *)(Q + (size_t)n * n);         // [2][c[half], s[half]] (n even: 8-byte aligned)
    int *perm = (int *)(csb + 2 * n);                    // n
    unsigned char *sched = (unsigned char *)(perm + n);  // (n - 1) x n players
    unsigned char *pqb = sched + (size_t)(n - 1) * n;    // [2][p[half], q[half]]
    __shared__ int s_any;
    __shared__ double s_red[32];
    __shared__ double s_first_off;
    const int k = blockIdx.x;
    const double live_floor = live_floor_ptr ? *live_floor_ptr : 0.0;
    const int half = n / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const float *g_in = Gin + (size_t)k * n * n;
    for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
        const int c = i / n, r = i - c * n;
        // symmetrise (the tensor-core Gram is symmetric up to rounding)
        G[i] = 0.5 * ((double)g_in[i] + (double)g_in[(size_t)r * n + c]);
        Q[i] = (r == c) ? 1.f : 0.f;
    }
    for (int i = threadIdx.x; i < (n - 1) * n; i += blockDim.x) {
        const int r = i / n, pos = i - r * n;
        sched[i] = (unsigned char)circ(pos, r, n);
    }
    if (threadIdx.x == 0) s_first_off = 0.0;
    __syncthreads();
    double dmax = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) dmax = fmax(dmax, G[(size_t)i * n + i]);
    for (int o = 16; o; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if (lane == 0) s_red[warp] = dmax;
    __syncthreads();
    double gmax = 0.0;
    for (int w = 0; w < nwarps; ++w) gmax = fmax(gmax, s_red[w]);
    const double floor_ = 2.220446049250313e-16 * 2.220446049250313e-16 * gmax;
    const double tol2 = tol * tol;
    int sweep = 0;
    for (sweep = 1; sweep <= max_sweeps; ++sweep) {
        __syncthreads();                                 // s_any readers of the last sweep are done
        if (threadIdx.x == 0) s_any = 0;
        // largest ratio^2 of the sweep as num / den (one division at the end)
        double offn = 0.0, offd = 1.0;
        for (int r = 0; r < n - 1; ++r) {
            const int buf = r & 1;
            double *cs = csb + buf * n;
            unsigned char *pq = pqb + buf * n;
            __syncthreads();                             // G of round r - 1 complete
            if (warp == 0) {
                for (int t = lane; t < half; t += 32) {
                    int p = sched[r * n + t], q = sched[r * n + n - 1 - t];
                    if (p > q) { const int x = p; p = q; q = x; }
                    const double app = G[p * n + p], aqq = G[q * n + q], apq = G[q * n + p];
                    double c = 1.0, sn = 0.0;
                    const double prod = app * aqq, apq2 = apq * apq;
                    if (apq2 > tol2 * prod && fmin(app, aqq) > floor_) {
                        // off over live columns only (norm^2 above live_floor),
                        // like the reference's convergence check (solvers.py:55-57)
                        if (fmin(app, aqq) > live_floor && apq2 * offd > offn * prod) { offn = apq2; offd = prod; }
                        const double d = aqq - app, a2 = 2.0 * fabs(apq);
                        // exact power-of-two scaling of (d, 2|apq|) into [1, 2) for the FP32 angle
                        const int ex = (__double2hiint(fmax(fabs(d), a2)) >> 20) & 0x7ff;
                        const double sc = __hiloint2double((2046 - ex) << 20, 0);
                        const float df = fabsf((float)(d * sc)), af = (float)(a2 * sc);
                        const float tf = __fdividef(af, df + sqrtf(df * df + af * af));
                        const double tt = d < 0.0 ? -(double)tf : (double)tf;
                        c = rsqrt(1.0 + tt * tt);
                        sn = tt * c;
                        if (apq < 0.0) sn = -sn;
                        s_any = 1;
                    }
                    cs[t] = c;
                    cs[half + t] = sn;
                    pq[t] = (unsigned char)p;
                    pq[half + t] = (unsigned char)q;
                }
            } else if (r > 0) {
                rotate_q(Q, pqb + (buf ^ 1) * n, csb + (buf ^ 1) * n, n, half, warp - 1, nwarps - 1, lane);
            }
            __syncthreads();
            // G <- J^T G J: warp w takes column pairs b = w, w + nwarps, ...,
            // its lanes the row pairs a (one 2 x 2 block per (a, b)).
            for (int b = warp; b < half; b += nwarps) {
                const int u = pq[b], v = pq[half + b];
                const double cb = cs[b], sb = cs[half + b];
                double *cu = G + u * n, *cv = G + v * n;
                for (int a = lane; a < half; a += 32) {
                    const int p = pq[a], q = pq[half + a];
                    const double ca = cs[a], sa = cs[half + a];
                    const double gpu = cu[p], gqu = cu[q], gpv = cv[p], gqv = cv[q];
                    // rows: [p; q] <- J_a^T [p; q] with J = [[c, s], [-s, c]] acting on columns (p, q)
                    const double rpu = ca * gpu - sa * gqu, rqu = sa * gpu + ca * gqu;
                    const double rpv = ca * gpv - sa * gqv, rqv = sa * gpv + ca * gqv;
                    // columns: [u, v] <- [u, v] J_b
                    cu[p] = cb * rpu - sb * rpv;
                    cv[p] = sb * rpu + cb * rpv;
                    cu[q] = cb * rqu - sb * rqv;
                    cv[q] = sb * rqu + cb * rqv;
                }
            }
        }
        // the last round's Q rotation, all warps
        rotate_q(Q, pqb + ((n - 2) & 1) * n, csb + ((n - 2) & 1) * n, n, half, warp, nwarps, lane);
        if (sweep == 1 && warp == 0) {
            for (int o = 16; o; o >>= 1) {
                const double on = __shfl_xor_sync(0xffffffffu, offn, o), od = __shfl_xor_sync(0xffffffffu, offd, o);
                if (on * offd > offn * od) { offn = on; offd = od; }
            }
            if (lane == 0) s_first_off = sqrt(offn / offd);
        }
        __syncthreads();
        if (!s_any) break;
    }
    __syncthreads();
    // Eigenvalues descending (stable), Q^T rows in that order.
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double dj = G[(size_t)j * n + j];
        int rk = 0;
        for (int i = 0; i < n; ++i) {
            const double di = G[(size_t)i * n + i];
            rk += (di > dj) || (di == dj && i < j);
        }
        perm[rk] = j;
    }
    __syncthreads();
    __nv_bfloat16 *qh = Qt_hi + (size_t)k * n * n, *ql = Qt_lo + (size_t)k * n * n;
    for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
        const int rrow = t / n, i = t - rrow * n;       // Q^T row rrow = column perm[rrow] of Q
        const float x = Q[(size_t)perm[rrow] * n + i];
        const __nv_bfloat16 h = __float2bfloat16_rn(x);
        qh[t] = h;
        const float rem = x - __bfloat162float(h);
        const __nv_bfloat16 l = __float2bfloat16_rn(rem);
        ql[t] = l;
        if (Qt_lo2) Qt_lo2[(size_t)k * n * n + t] = __float2bfloat16_rn(rem - __bfloat162float(l));
    }
    if (threadIdx.x == 0) {
        if (off_out) off_out[k] = (float)s_first_off;
        if (dmax_out) dmax_out[k] = (float)gmax;
        if (sweeps_out) sweeps_out[k] = sweep > max_sweeps ? max_sweeps : sweep;
    }
}

// Register-resident variant of eig_kernel for n = 32 * RPT (64 or 128), the
// slot widths of b = 32 and b = 64.  Same rotations and outputs; the pairs of
// a sweep follow the odd-even ordering instead of the round robin: round r
// pairs adjacent positions (2t + r % 2, 2t + r % 2 + 1) and every rotation
// also swaps its two positions (J P), so after n rounds each pair of columns
// has met exactly once (the swaps reverse the order).  With positions fixed,
// G and Q stay in registers: lane l holds rows RPT l .. RPT l + RPT - 1 and
// warp w columns CB w .. CB w + CB - 1 (CB even: 4, 8 or 16 columns per warp,
// n / CB warps; the outputs do not depend on CB).  Row pairs that straddle two
// lanes and column pairs that straddle two warps (odd rounds) are exchanged.
// Per round: the first warps form the angles from the diagonal d and
// superdiagonal e (published in shared memory by their owners), one barrier,
// rotations, (odd rounds: boundary exchange, one barrier), new d / e, one
// barrier.
// DQ (deferred Q): Q is not accumulated here.  The angle threads record every
// applied (c, s) as FP32 pairs, cs_out[(k * max_sweeps + sweep) * n + r][p]
// by the pair's first position p, and the kernel writes the eigenvalues'
// sorted position of every column (pos_out[k * n + j]); q_apply_kernel then
// forms Q^T from them on other SMs, so this latency-bound kernel issues
// about a quarter fewer instructions per round.
//
// FP32 G is scaled, G = D G_s D, and Q = Q_s D, with a scale per position (FP64):
// a rotation is then x + b y, y - a x with both scales multiplied by c, one
// multiply-add an element instead of two (Gentleman's rotation), and c = 1 -
// t^2 / (...) does not round the cosines of small angles to 1, always to the
// same side (||Q^T Q - I|| of two sweeps 2.4e-5 -> 2.2e-6).  Scales below 2^-8
// are multiplied in, once or twice in a sweep of a dense random G.  (FP64 G is
// not scaled: the scales' own chain costs what the shorter rotations give.)  Q
// lags one round: while the first warps form the angles of a round, the others
// apply the previous round's to their tiles of Q.  Rows and columns that cross
// a lane or a warp go through shared memory in 16-byte accesses (FP32: shuffles
// took three times as long; FP64 rows by shuffles).  One SM a slot, bound by
// the latency and the instruction issue of a round; two sweeps of n = 128, 8
// columns a warp: FP32 G 287 us, 383 with plain rotations, shuffles and Q
// rotated with G; FP64 G 534 (16 columns a warp), before 570.

// Bytes of the write-out area (n x n FP32) and of the boundary rows (512 a column), n <= 128.
__host__ __device__ constexpr size_t eig_reg_area_bytes(int n) { return (size_t)n * 512; }

template <typename TG> struct Pair2;
template <> struct Pair2<float> { using T = float2; };
template <> struct Pair2<double> { using T = double2; };

// N consecutive elements to and from shared memory in accesses of up to 16 bytes.
template <typename T, int N>
struct Run {
    static constexpr int B = (int)sizeof(T) * N, W = B % 16 == 0 ? 16 : B % 8 == 0 ? 8 : 4, C = W / (int)sizeof(T);
    struct alignas(W) Chunk { T v[C]; };
    __device__ static __forceinline__ void put(T *dst, const T (&v)[N]) {
#pragma unroll
        for (int i = 0; i < N / C; ++i) {
            Chunk c;
#pragma unroll
            for (int e = 0; e < C; ++e) c.v[e] = v[i * C + e];
            ((Chunk *)dst)[i] = c;
        }
    }
    __device__ static __forceinline__ void get(const T *src, T (&v)[N]) {
#pragma unroll
        for (int i = 0; i < N / C; ++i) {
            const Chunk c = ((const Chunk *)src)[i];
#pragma unroll
            for (int e = 0; e < C; ++e) v[i * C + e] = c.v[e];
        }
    }
};

// Tangent of a live, active pair, and the cosine of a tangent.
__device__ __forceinline__ float eig_tan(float app, float aqq, float apq) {
    // |zeta| <= 1e18 keeps its square finite (t is then below 1e-18)
    const float zeta = fminf(__fdividef(fabsf(aqq - app), 2.f * fabsf(apq)), 1e18f);
    const float h = fmaf(zeta, zeta, 1.f);
    const float t = __fdividef(1.f, zeta + h * rsqrtf(h));
    return (aqq < app) != (apq < 0.f) ? -t : t;
}
__device__ __forceinline__ double eig_tan(double app, double aqq, double apq) {
    const double d = aqq - app, a2 = 2.0 * fabs(apq);
    const int ex = (__double2hiint(fmax(fabs(d), a2)) >> 20) & 0x7ff;
    const double scl = __hiloint2double((2046 - ex) << 20, 0);
    const float df = fabsf((float)(d * scl)), af = (float)(a2 * scl);
    const float tf = __fdividef(af, df + sqrtf(df * df + af * af));
    return (d < 0.0) != (apq < 0.0) ? -(double)tf : (double)tf;
}
__device__ __forceinline__ double eig_cos(float t) { return cosine(t * t); }
__device__ __forceinline__ double eig_cos(double t) {        // FP32 estimate and one Newton step in FP64
    const double x = 1.0 + t * t, c0 = (double)rsqrtf(1.f + (float)t * (float)t);
    return c0 * (1.5 - 0.5 * x * c0 * c0);
}

template <int RPT, int CB, typename TG, bool DQ = false>
__global__ void __launch_bounds__(RPT * 1024 / CB) eig_reg_kernel(const float *Gin, __nv_bfloat16 *Qt_hi,
                                                            __nv_bfloat16 *Qt_lo, __nv_bfloat16 *Qt_lo2,
                                                            float *off_out, float *dmax_out, int *sweeps_out,
                                                            int max_sweeps, double tol, const double *live_floor_ptr,
                                                            float2 *cs_out, int *pos_out) {
    constexpr int n = 32 * RPT;
    constexpr int NW = n / CB, AW = RPT / 2;   // warps; those that form the angles (the next AW the scales)
    constexpr bool SC = sizeof(TG) == 4;       // scaled
    using T2 = typename Pair2<TG>::T;
    static_assert(CB % 2 == 0 && NW >= 2 * AW && RPT % 2 == 0, "columns per warp");
    extern __shared__ __align__(16) unsigned char smem[];
    double *scl = (double *)smem;              // scale of position x
    T2 *sab = (T2 *)(scl + n);                 // [2][n] (a, b) of the pair starting at position p, at cs_at(p)
    TG *sd = (TG *)(sab + 2 * n);              // d[x] = G_s[x][x]
    TG *se = sd + n;                           // e[x] = G_s[x][x + 1]
    T2 *sfi = (T2 *)(se + n);                  // the scale of position x and its inverse
    TG *st = (TG *)(sfi + n);                  // tangent of pair t
    TG *bg = st + n;                           // [NW][2][32][RPT] boundary columns of G (first, last)
    float *bq = (float *)(bg + (size_t)NW * 2 * n);  // [NW][2][32][RPT] boundary columns of Q
    float *Qs = bq + (size_t)NW * 2 * n;       // n x n, Q[col * n + row] (write-out)
    TG *br = (TG *)Qs;                         // [NW][2][CB / chunk][32][chunk] boundary rows of G (before the write-out)
    int *perm = (int *)((unsigned char *)Qs + eig_reg_area_bytes(n));   // n
    __shared__ int s_any, s_small;
    __shared__ double s_first_off;
    __shared__ double s_red[NW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = lane * RPT, c0 = warp * CB;
    // Shared-memory slots of per-row data, lane-major: row x = RPT l + i (lane l's i-th row) at
    // 32 i + l, so that the 32 lanes reading "their" i-th row hit 32 consecutive words instead of
    // one bank RPT-fold; a warp-uniform row is a broadcast either way.
    auto cs_at = [](int x) { return (x % RPT) * 32 + x / RPT; };
    auto bnd_at = [](int w, int side, int l) { return ((w * 2 + side) * 32 + l) * RPT; };
    const int k = blockIdx.x;
    const double live_floor = live_floor_ptr ? *live_floor_ptr : 0.0;
    const float *g_in = Gin + (size_t)k * n * n;

    TG g[RPT][CB];
    float2 q[RPT / 2][CB];                     // rows 2 i and 2 i + 1 of Q's tile
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int j = 0; j < CB; ++j) {
            const int r = r0 + i, c = c0 + j;
            // symmetrise (the tensor-core Gram is symmetric up to rounding)
            g[i][j] = (TG)(0.5 * ((double)g_in[(size_t)r * n + c] + (double)g_in[(size_t)c * n + r]));
            if (i & 1) q[i / 2][j].y = (r == c) ? 1.f : 0.f;
            else q[i / 2][j].x = (r == c) ? 1.f : 0.f;
        }
    // d and e: rows r0.. of a lane meet this warp's columns in LB lanes (both),
    // and in the lane before them (the e of its last row)
    constexpr int LB = CB / RPT > 0 ? CB / RPT : 1;
    static_assert(CB % RPT == 0 || RPT % CB == 0, "tiles");
    auto publish_de = [&]() {
        if constexpr (CB >= RPT) {
#pragma unroll
            for (int b = 0; b < LB; ++b)
                if (lane == warp * LB + b) {
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        sd[r0 + i] = g[i][b * RPT + i];
                        if (b * RPT + i + 1 < CB) se[r0 + i] = g[i][b * RPT + i + 1];
                    }
                }
            if (lane == warp * LB - 1) se[r0 + RPT - 1] = g[RPT - 1][0];
        } else {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    if (c0 + j == r0 + i) sd[r0 + i] = g[i][j];
                    if (c0 + j == r0 + i + 1) se[r0 + i] = g[i][j];
                }
        }
    };
    // A rotation and the swap of its positions, x, y <- first(x, y), second(y, x):
    // y + b x and x - a y of (a, b) when scaled, else s x + c y and c x - s y of (s, c).
    // (the larger product inside the multiply-add)
    auto first = [](TG own, TG other, T2 v) -> TG { return SC ? fma(v.y, own, other) : fma(v.y, other, v.x * own); };
    auto second = [](TG own, TG other, T2 v) -> TG { return SC ? fma(-v.x, own, other) : fma(v.y, other, -v.x * own); };
    auto turn = [&](TG &x, TG &y, T2 v) {
        const TG u = x;
        x = first(u, y, v);
        y = second(y, u, v);
    };
    auto both = [](float v) { return make_float2(v, v); };
    auto first_q = [&](float2 own, float2 other, T2 v) {
        if constexpr (SC) return __ffma2_rn(both(v.y), own, other);
        else return __ffma2_rn(both((float)v.y), other, __fmul2_rn(both((float)v.x), own));
    };
    auto second_q = [&](float2 own, float2 other, T2 v) {
        if constexpr (SC) return __ffma2_rn(both(-v.x), own, other);
        else return __ffma2_rn(both((float)v.y), other, __fmul2_rn(both(-(float)v.x), own));
    };
    auto turn_q = [&](float2 &x, float2 &y, T2 v) {
        const float2 u = x;
        x = first_q(u, y, v);
        y = second_q(y, u, v);
    };
    // Q's column rotations of a round of parity par with the angles of buffer buf
    auto update_q = [&](int par, int buf) {
        const T2 *ab = sab + buf * n;
        if (par == 0) {
#pragma unroll
            for (int j = 0; j < CB; j += 2) {
                const T2 t = ab[cs_at(c0 + j)];
#pragma unroll
                for (int i = 0; i < RPT / 2; ++i) turn_q(q[i][j], q[i][j + 1], t);
            }
        } else {
            if (warp > 0) {                    // pair (c0 - 1, c0): this warp holds the second
                const T2 v = ab[cs_at(c0 - 1)];
                float x[RPT];
                Run<float, RPT>::get(bq + bnd_at(warp - 1, 1, lane), x);
#pragma unroll
                for (int i = 0; i < RPT / 2; ++i)
                    q[i][0] = second_q(q[i][0], make_float2(x[2 * i], x[2 * i + 1]), v);
            }
            if (warp < NW - 1) {               // pair (c0 + CB - 1, c0 + CB): this warp holds the first
                const T2 v = ab[cs_at(c0 + CB - 1)];
                float y[RPT];
                Run<float, RPT>::get(bq + bnd_at(warp + 1, 0, lane), y);
#pragma unroll
                for (int i = 0; i < RPT / 2; ++i)
                    q[i][CB - 1] = first_q(q[i][CB - 1], make_float2(y[2 * i], y[2 * i + 1]), v);
            }
#pragma unroll
            for (int j = 1; j + 1 < CB; j += 2) {
                const T2 t = ab[cs_at(c0 + j)];
#pragma unroll
                for (int i = 0; i < RPT / 2; ++i) turn_q(q[i][j], q[i][j + 1], t);
            }
        }
    };
    publish_de();
    T2 one;
    one.x = one.y = (TG)1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        scl[i] = 1.0;
        sfi[i] = one;
    }
    if (threadIdx.x == 0) { s_first_off = 0.0; s_small = 0; }
    __syncthreads();
    double dm = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) dm = fmax(dm, (double)sd[i]);
    for (int o = 16; o; o >>= 1) dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
    if (lane == 0) s_red[warp] = dm;
    __syncthreads();
    double gmax = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) gmax = fmax(gmax, s_red[w]);
    // eps of the arithmetic squared times the largest diagonal: the active floor
    constexpr double eps_g = sizeof(TG) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-07;
    const TG floor_ = (TG)(eps_g * eps_g * gmax), live = (TG)live_floor;
    const TG tol2 = (TG)(tol * tol);
    int sweep = 0, buf = 0;                    // buf: the angles of the round at hand
    bool lag = false;                          // Q still lacks the previous round (odd, or even: its parity is 1 - par)
    for (sweep = 1; sweep <= max_sweeps; ++sweep) {
        if (threadIdx.x == 0) s_any = 0;
        TG offm = 0;                           // the largest a_pq^2 / (a_pp a_qq) this thread met
        for (int r = 0; r < n; ++r, buf ^= 1) {
            const int par = r & 1;
            __syncthreads();                   // d / e of the previous round published; s_any reset
            const bool small = s_small != 0;
            if (warp < AW) {                   // the angles, a pair a lane
                const int p = 2 * threadIdx.x + par;
                if (p + 1 < n) {
                    T2 fp, fq;
                    TG app = sd[p], aqq = sd[p + 1], apq = se[p];
                    if constexpr (SC) {
                        fp = sfi[p];
                        fq = sfi[p + 1];
                        app *= fp.x * fp.x;
                        aqq *= fq.x * fq.x;
                        apq *= fp.x * fq.x;
                    }
                    const TG low = app < aqq ? app : aqq;
                    bool on;
                    TG ratio = 0, tt = 0;
                    if constexpr (sizeof(TG) == 4) {         // no product of two small entries: no underflow
                        ratio = low > floor_ ? __fdividef(apq, app) * __fdividef(apq, aqq) : 0.f;
                        on = ratio > tol2;
                    } else {
                        on = apq * apq > tol2 * (app * aqq) && low > floor_;
                        if (on && sweep == 1) ratio = apq * apq / (app * aqq);
                    }
                    if (on) {
                        // off over live columns only (solvers.py:55-57)
                        if (low > live && ratio > offm) offm = ratio;
                        tt = eig_tan(app, aqq, apq);
                        s_any = 1;
                    }
                    T2 v;
                    if constexpr (SC) {
                        v.x = tt * (fq.x * fp.y);
                        v.y = tt * (fp.x * fq.y);
                        st[threadIdx.x] = tt;
                    } else {
                        v.y = on ? eig_cos(tt) : (TG)1;
                        v.x = tt * v.y;
                        if constexpr (DQ)
                            cs_out[(((size_t)k * max_sweeps + (sweep - 1)) * n + r) * n + p] =
                                make_float2((float)v.y, (float)v.x);
                    }
                    sab[buf * n + cs_at(p)] = v;
                }
            } else if constexpr (!DQ) {
                if (lag) update_q(1 - par, buf ^ 1);
            }
            __syncthreads();
            const T2 *ab = sab + buf * n;
            if (warp < AW) {
                if constexpr (!DQ)
                    if (lag) update_q(1 - par, buf ^ 1);
            } else if (SC && warp < 2 * AW) {  // the scales, which the next round's angles need
                const int x = threadIdx.x - 32 * AW, p = 2 * x + par;
                if (p + 1 < n) {
                    const TG tt = st[x];
                    const double c = eig_cos(tt), np_ = c * scl[p + 1], nq_ = c * scl[p];
                    T2 f, h;
                    f.x = (TG)np_;
                    f.y = inv_scale(f.x);
                    h.x = (TG)nq_;
                    h.y = inv_scale(h.x);
                    scl[p] = np_;
                    scl[p + 1] = nq_;
                    sfi[p] = f;
                    sfi[p + 1] = h;
                    if (fmin(np_, nq_) < 0.00390625) s_small = 1;
                    if constexpr (DQ)
                        cs_out[(((size_t)k * max_sweeps + (sweep - 1)) * n + r) * n + p] =
                            make_float2((float)c, (float)((double)tt * c));
                }
            }
            // Rows (J^T from the left, then the swap).
            if (par == 0) {
#pragma unroll
                for (int i = 0; i < RPT; i += 2) {
                    const T2 v = ab[32 * i + lane];          // pair at row r0 + i
#pragma unroll
                    for (int j = 0; j < CB; ++j) turn(g[i][j], g[i + 1][j], v);
                }
            } else {
                // pairs at rows r0 - 1 (lane - 1's last row) and r0 + RPT - 1 (this lane's last row);
                // their other rows through shared memory (FP32) or by shuffles
                constexpr int CH = 16 / (int)sizeof(TG) < CB ? 16 / (int)sizeof(TG) : CB;
                TG *mine = br + (size_t)warp * 2 * CB * 32 + lane * CH;
                if constexpr (SC) {
#pragma unroll
                    for (int jc = 0; jc < CB / CH; ++jc) {
                        TG f[CH], l[CH];
#pragma unroll
                        for (int e = 0; e < CH; ++e) {
                            f[e] = g[0][jc * CH + e];
                            l[e] = g[RPT - 1][jc * CH + e];
                        }
                        Run<TG, CH>::put(mine + jc * 32 * CH, f);
                        Run<TG, CH>::put(mine + (CB / CH + jc) * 32 * CH, l);
                    }
                    __syncwarp();
                }
                const int up = lane > 0 ? -CH : 0, down = lane < 31 ? CH : 0;
                T2 vu, vd;                     // no pair: the row itself, from a zero other row
                vu.x = (TG)-1;
                vu.y = (TG)0;
                vd.x = vd.y = (TG)1;
                if constexpr (!SC) vd.y = (TG)0;
                if (lane > 0) vu = ab[32 * (RPT - 1) + lane - 1];
                if (lane < 31) vd = ab[32 * (RPT - 1) + lane];
                if constexpr (SC) {
#pragma unroll
                    for (int jc = 0; jc < CB / CH; ++jc) {
                        TG f[CH], l[CH];
                        Run<TG, CH>::get(mine + (CB / CH + jc) * 32 * CH + up, l);
                        Run<TG, CH>::get(mine + jc * 32 * CH + down, f);
#pragma unroll
                        for (int e = 0; e < CH; ++e) {
                            const int j = jc * CH + e;
                            g[0][j] = second(g[0][j], lane > 0 ? l[e] : (TG)0, vu);
                            g[RPT - 1][j] = first(g[RPT - 1][j], lane < 31 ? f[e] : (TG)0, vd);
                        }
                    }
                    __syncwarp();
                } else {
#pragma unroll
                    for (int j = 0; j < CB; ++j) {
                        const TG l = __shfl_up_sync(0xffffffffu, g[RPT - 1][j], 1);      // row r0 - 1
                        const TG f = __shfl_down_sync(0xffffffffu, g[0][j], 1);          // row r0 + RPT
                        g[0][j] = second(g[0][j], lane > 0 ? l : (TG)0, vu);
                        g[RPT - 1][j] = first(g[RPT - 1][j], lane < 31 ? f : (TG)0, vd);
                    }
                }
#pragma unroll
                for (int i = 1; i + 1 < RPT; i += 2) {
                    const T2 v = ab[32 * i + lane];          // pair at row r0 + i
#pragma unroll
                    for (int j = 0; j < CB; ++j) turn(g[i][j], g[i + 1][j], v);
                }
            }
            // Columns (J from the right, then the swap).
            if (par == 0) {
#pragma unroll
                for (int j = 0; j < CB; j += 2) {
                    const T2 v = ab[cs_at(c0 + j)];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) turn(g[i][j], g[i][j + 1], v);
                }
            } else {
                // publish this warp's first and last columns (G after the row rotation, Q for update_q)
                TG lo[RPT], hi[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    lo[i] = g[i][0];
                    hi[i] = g[i][CB - 1];
                }
                Run<TG, RPT>::put(bg + bnd_at(warp, 0, lane), lo);
                Run<TG, RPT>::put(bg + bnd_at(warp, 1, lane), hi);
                if constexpr (!DQ) {
                    float qf[RPT], ql[RPT];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        qf[i] = i & 1 ? q[i / 2][0].y : q[i / 2][0].x;
                        ql[i] = i & 1 ? q[i / 2][CB - 1].y : q[i / 2][CB - 1].x;
                    }
                    Run<float, RPT>::put(bq + bnd_at(warp, 0, lane), qf);
                    Run<float, RPT>::put(bq + bnd_at(warp, 1, lane), ql);
                }
                __syncthreads();
                if (warp > 0) {                // pair (c0 - 1, c0): this warp holds the second
                    const T2 v = ab[cs_at(c0 - 1)];
                    Run<TG, RPT>::get(bg + bnd_at(warp - 1, 1, lane), hi);
#pragma unroll
                    for (int i = 0; i < RPT; ++i) g[i][0] = second(g[i][0], hi[i], v);
                }
                if (warp < NW - 1) {           // pair (c0 + CB - 1, c0 + CB): this warp holds the first
                    const T2 v = ab[cs_at(c0 + CB - 1)];
                    Run<TG, RPT>::get(bg + bnd_at(warp + 1, 0, lane), lo);
#pragma unroll
                    for (int i = 0; i < RPT; ++i) g[i][CB - 1] = first(g[i][CB - 1], lo[i], v);
                }
#pragma unroll
                for (int j = 1; j + 1 < CB; j += 2) {
                    const T2 v = ab[cs_at(c0 + j)];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) turn(g[i][j], g[i][j + 1], v);
                }
            }
            lag = true;
            if (SC && small) {                       // read after the round's first barrier: the same in every thread
                if constexpr (!DQ) update_q(par, buf);
                lag = false;
                __syncthreads();
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    const double dj = scl[c0 + j];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) g[i][j] *= (TG)(scl[r0 + i] * dj);
#pragma unroll
                    for (int i = 0; i < RPT / 2; ++i) {
                        q[i][j].x *= (float)dj;
                        q[i][j].y *= (float)dj;
                    }
                }
                __syncthreads();
                for (int i = threadIdx.x; i < n; i += blockDim.x) {
                    scl[i] = 1.0;
                    sfi[i] = one;
                }
                if (threadIdx.x == 0) s_small = 0;
            }
            publish_de();
        }
        if (sweep == 1 && warp < AW) {
            for (int o = 16; o; o >>= 1) {
                const TG v = __shfl_xor_sync(0xffffffffu, offm, o);
                offm = v > offm ? v : offm;
            }
            if (lane == 0) s_red[warp] = sqrt((double)offm);
        }
        __syncthreads();
        if (sweep == 1 && threadIdx.x == 0) {
            double o = 0.0;
#pragma unroll
            for (int w = 0; w < AW; ++w) o = fmax(o, s_red[w]);
            s_first_off = o;
        }
        const int any = s_any;
        __syncthreads();                       // everyone has read s_any before it is reset
        if (!any) break;
    }
    if constexpr (!DQ)
        if (lag) update_q(1, buf ^ 1);         // a sweep ends on an odd round
    // Q to shared memory (column-major) for the sorted write-out; scales back in.
    if constexpr (!DQ) {
#pragma unroll
        for (int j = 0; j < CB; ++j) {
            const double dj = scl[c0 + j];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                Qs[(size_t)(c0 + j) * n + r0 + i] = (float)(dj * (double)(i & 1 ? q[i / 2][j].y : q[i / 2][j].x));
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) sd[i] = (TG)((double)sd[i] * scl[i] * scl[i]);
    __syncthreads();
    // Eigenvalues descending (stable), Q^T rows in that order.
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double dj = sd[j];
        int rk = 0;
        for (int i = 0; i < n; ++i) {
            const double di = sd[i];
            rk += (di > dj) || (di == dj && i < j);
        }
        perm[rk] = j;
        if constexpr (DQ) pos_out[(size_t)k * n + j] = rk;
    }
    __syncthreads();
    __nv_bfloat16 *qh = Qt_hi + (size_t)k * n * n, *ql = Qt_lo + (size_t)k * n * n;
    for (int t = threadIdx.x; t < (DQ ? 0 : n * n); t += blockDim.x) {
        const int rrow = t / n, i = t - rrow * n;       // Q^T row rrow = column perm[rrow] of Q
        const float x = Qs[(size_t)perm[rrow] * n + i];
        const __nv_bfloat16 h = __float2bfloat16_rn(x);
        qh[t] = h;
        const float rem = x - __bfloat162float(h);
        const __nv_bfloat16 l = __float2bfloat16_rn(rem);
        ql[t] = l;
        if (Qt_lo2) Qt_lo2[(size_t)k * n * n + t] = __float2bfloat16_rn(rem - __bfloat162float(l));
    }
    if (threadIdx.x == 0) {
        if (off_out) off_out[k] = (float)s_first_off;
        if (dmax_out) dmax_out[k] = (float)gmax;
        if (sweeps_out) sweeps_out[k] = sweep > max_sweeps ? max_sweeps : sweep;
    }
}

// Q^T of every slot from the rotations eig_reg_kernel<..., DQ = true>
// recorded.  Warp (k, i) forms row i of Q = prod_r J_r P_r with the same FP32
// column updates the register kernel applies to its Q tiles (lane l holds
// columns RPT l .. RPT l + RPT - 1; in odd rounds the pairs that straddle two
// lanes take the neighbour's value by a shuffle), then writes it as column i
// of Q^T in eigenvalue order (row pos[j] for column j), as hi / lo (/ lo2)
// BF16 parts.  Rows are independent, so the whole grid works at once.
template <int RPT>
__global__ void __launch_bounds__(256) q_apply_kernel(const float2 *cs, const int *sweeps, const int *pos,
                                                      __nv_bfloat16 *Qt_hi, __nv_bfloat16 *Qt_lo,
                                                      __nv_bfloat16 *Qt_lo2, int pairs, int max_sweeps) {
    constexpr int n = 32 * RPT;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= (int64_t)pairs * n) return;                  // whole warps
    const int k = (int)(gw / n), i = (int)(gw - (int64_t)k * n);
    const int c0 = lane * RPT;
    float q[RPT];
#pragma unroll
    for (int e = 0; e < RPT; ++e) q[e] = (c0 + e == i) ? 1.f : 0.f;
    int ns = sweeps[k];
    if (ns > max_sweeps) ns = max_sweeps;
    const float2 *ck = cs + (size_t)k * max_sweeps * n * n;
    for (int rr = 0; rr < ns * n; ++rr) {
        const float2 *c_r = ck + (size_t)rr * n;
        if ((rr & 1) == 0) {
#pragma unroll
            for (int e = 0; e < RPT; e += 2) {
                const float2 t = c_r[c0 + e];
                const float u = q[e], v = q[e + 1];
                q[e] = t.y * u + t.x * v;
                q[e + 1] = t.x * u - t.y * v;
            }
        } else {
            const bool has_up = lane > 0, has_down = lane < 31;
            const float2 tu = has_up ? c_r[c0 - 1] : make_float2(1.f, 0.f);
            const float2 td = has_down ? c_r[c0 + RPT - 1] : make_float2(1.f, 0.f);
            const float up = __shfl_up_sync(0xffffffffu, q[RPT - 1], 1);    // column c0 - 1
            const float dn = __shfl_down_sync(0xffffffffu, q[0], 1);        // column c0 + RPT
            const float first = q[0], last = q[RPT - 1];
            if (has_up) q[0] = tu.x * up - tu.y * first;                      // second of (c0 - 1, c0)
            if (has_down) q[RPT - 1] = td.y * last + td.x * dn;               // first of (c0 + RPT - 1, c0 + RPT)
#pragma unroll
            for (int e = 1; e + 1 < RPT; e += 2) {
                const float2 t = c_r[c0 + e];
                const float u = q[e], v = q[e + 1];
                q[e] = t.y * u + t.x * v;
                q[e + 1] = t.x * u - t.y * v;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < RPT; ++e) {
        const size_t t = (size_t)k * n * n + (size_t)pos[(size_t)k * n + c0 + e] * n + i;
        const float x = q[e];
        const __nv_bfloat16 h = __float2bfloat16_rn(x);
        Qt_hi[t] = h;
        const float rem = x - __bfloat162float(h);
        const __nv_bfloat16 l = __float2bfloat16_rn(rem);
        Qt_lo[t] = l;
        if (Qt_lo2) Qt_lo2[t] = __float2bfloat16_rn(rem - __bfloat162float(l));
    }
}

__host__ inline size_t eig_reg_smem_bytes(int n, int cb) {   // sized for FP64 G (enough for FP32)
    const int nw = n / cb;
    return (size_t)10 * n * 8 + (size_t)nw * 2 * n * 8 + (size_t)nw * 2 * n * 4 + eig_reg_area_bytes(n) +
           (size_t)n * 4 + 16;
}

// dst row map[r] <- src row r (length L), split into hi / lo BF16.
__global__ void scatter_kernel(const float *src, const int *map, __nv_bfloat16 *hi, __nv_bfloat16 *lo,
                               __nv_bfloat16 *lo2, float *f32, int64_t rows, int64_t L) {
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
        const int64_t d = map ? map[r] : r;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < L; i += (int64_t)gridDim.x * blockDim.x) {
            const float v = src[r * L + i];
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            if (hi) hi[d * L + i] = h;
            const float rem = v - __bfloat162float(h);
            const __nv_bfloat16 l = __float2bfloat16_rn(rem);
            if (lo) lo[d * L + i] = l;
            if (lo2) lo2[d * L + i] = __float2bfloat16_rn(rem - __bfloat162float(l));
            if (f32) f32[d * L + i] = v;
        }
    }
}

__global__ void combine_kernel(const __nv_bfloat16 *hi, const __nv_bfloat16 *lo, const __nv_bfloat16 *lo2,
                               const int *map, float *dst, int64_t rows, int64_t L) {
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
        const int64_t d = map ? map[r] : r;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < L; i += (int64_t)gridDim.x * blockDim.x)
            dst[d * L + i] = __bfloat162float(hi[r * L + i]) + (lo ? __bfloat162float(lo[r * L + i]) : 0.f) +
                             (lo2 ? __bfloat162float(lo2[r * L + i]) : 0.f);
    }
}

// sigma_j = ||Wt row j|| * 2^e (FP64 sums), one warp per row.
__global__ void norms_kernel(const float *Wt, double *sig, int64_t n, int64_t m) {
    const int64_t row = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    double acc = 0.0;
    for (int64_t i = lane; i < m; i += 32) {
        const double x = Wt[row * m + i];
        acc = fma(x, x, acc);
    }
    acc = warp_sum_d(acc);
    if (lane == 0) sig[row] = sqrt(acc);
}

// Stable descending rank of every sigma (n^2 comparisons, n <= a few 1000).
__global__ void rank_kernel(const double *sig, int *perm, int n) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double sj = sig[j];
    int rk = 0;
    for (int i = 0; i < n; ++i) {
        const double si = sig[i];
        rk += (si > sj) || (si == sj && i < j);
    }
    perm[rk] = j;
}

// Outputs: S[r] (cut below eps32 max(m, n_even) sigma_1), U[:, r] = W_perm[r] /
// sigma (kept columns; cut columns of nonzero norm are normalised the same
// way), Vh[r, :] = Vt[perm[r], :].
__global__ void finish_kernel(const float *Wt, const float *Vt, const double *sig, const int *perm, float *U,
                              float *S, float *Vh, int64_t m, int64_t n, int rank, int e, int cutw) {
    const double smax = sig[perm[0]];
    const double cut = 1.1920928955078125e-07 * (double)cutw * smax;
    const int64_t total_u = m * rank, total_v = (int64_t)rank * n;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total_u + total_v + rank;
         t += (int64_t)gridDim.x * blockDim.x) {
        if (t < total_u) {
            const int64_t i = t / rank, r = t - i * rank;
            const int j = perm[r];
            const double sj = sig[j];
            U[t] = U ? (float)(sj > 0.0 ? Wt[(int64_t)j * m + i] / sj : 0.0) : 0.f;
        } else if (t < total_u + total_v) {
            const int64_t q = t - total_u, r = q / n, c = q - r * n;
            Vh[q] = Vt[(int64_t)perm[r] * n + c];
        } else {
            const int r = (int)(t - total_u - total_v);
            const double sj = sig[perm[r]];
            S[r] = (float)(sj > cut ? ldexp(sj, e) : 0.0);
        }
    }
}


// C (M x N, f32) = A (M x K) * B (N x K)^T with FP32 inputs (row-major, K
// contiguous) and FP64 accumulation: every product of two floats is exact in
// FP64, so C carries FP64 accuracy until its final rounding.  128 x 128
// tiles, K steps of 8, 256 threads with 8 x 8 outputs each.
__global__ void __launch_bounds__(256) gemm_f64acc_kernel(const float *A, const float *B, float *C, int64_t M,
                                                          int64_t N, int64_t K, int64_t lda, int64_t ldb,
                                                          int64_t ldc) {
    __shared__ double As[8][128];
    __shared__ double Bs[8][128];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int64_t m0 = (int64_t)blockIdx.y * 128, n0 = (int64_t)blockIdx.x * 128;
    double acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    const int lr = threadIdx.x >> 1, lk = (threadIdx.x & 1) * 4;
    for (int64_t k0 = 0; k0 < K; k0 += 8) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int64_t ka = k0 + lk + q;
            const int64_t ra = m0 + lr, rb = n0 + lr;
            As[lk + q][lr] = (ra < M && ka < K) ? (double)A[ra * lda + ka] : 0.0;
            Bs[lk + q][lr] = (rb < N && ka < K) ? (double)B[rb * ldb + ka] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            double a[8], b[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = As[k][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t r = m0 + ty + 16 * i;
        if (r >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int64_t c = n0 + tx + 16 * j;
            if (c < N) C[r * ldc + c] = (float)acc[i][j];
        }
    }
}

// The same product for 16-byte aligned rows (A, B 16-byte aligned; lda, ldb
// and K multiples of 4): the next 16-deep K slice is fetched with float4
// loads into registers while the current slice's FMAs run, then stored as
// FP64 into the other half of a double-buffered shared tile, so each slice
// costs one barrier and no exposed global latency.  Thread (ty, tx) owns rows
// 2 ty + 32 i + {0, 1} and columns 2 tx + 32 j + {0, 1} (i, j < 4): its
// operands are double2 loads from shared memory.
constexpr int kF64KC = 16;
constexpr size_t kF64AccSmem = 2 * 2 * kF64KC * 128 * sizeof(double);   // [A, B][2][16][128]

__global__ void __launch_bounds__(256) gemm_f64acc_vec_kernel(const float *A, const float *B, float *C, int64_t M,
                                                              int64_t N, int64_t K, int64_t lda, int64_t ldb,
                                                              int64_t ldc, int m_fast) {
    extern __shared__ __align__(16) double f64acc_smem[];
    double *As = f64acc_smem;                      // As[buf][k][row] at (buf * kF64KC + k) * 128 + row
    double *Bs = f64acc_smem + 2 * kF64KC * 128;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // m_fast: consecutive CTAs take consecutive row tiles of C, so the tile of
    // B (the larger operand) they share is read from DRAM once
    const int64_t m0 = (int64_t)(m_fast ? blockIdx.x : blockIdx.y) * 128,
                  n0 = (int64_t)(m_fast ? blockIdx.y : blockIdx.x) * 128;
    // loader: row lrow of the tile, K offsets lk and lk + 8 of the slice
    const int lrow = threadIdx.x & 127, lk = (threadIdx.x >> 7) * 4;
    const bool arow = m0 + lrow < M, brow = n0 + lrow < N;
    const float *ap = A + (arow ? (m0 + lrow) * lda : 0), *bp = B + (brow ? (n0 + lrow) * ldb : 0);
    float4 pa[2], pb[2];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const int64_t ka = k0 + lk + 8 * l;
            const bool kin = ka < K;               // K % 4 == 0: a float4 is wholly in or out
            pa[l] = (arow && kin) ? *(const float4 *)(ap + ka) : make_float4(0.f, 0.f, 0.f, 0.f);
            pb[l] = (brow && kin) ? *(const float4 *)(bp + ka) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            double *a = As + ((size_t)buf * kF64KC + lk + 8 * l) * 128 + lrow;
            double *b = Bs + ((size_t)buf * kF64KC + lk + 8 * l) * 128 + lrow;
            a[0] = pa[l].x; a[128] = pa[l].y; a[256] = pa[l].z; a[384] = pa[l].w;
            b[0] = pb[l].x; b[128] = pb[l].y; b[256] = pb[l].z; b[384] = pb[l].w;
        }
    };
    double acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    const int64_t nk = (K + kF64KC - 1) / kF64KC;
    fetch(0);
    stash(0);
    __syncthreads();
    for (int64_t kb = 0; kb < nk; ++kb) {
        const int buf = (int)(kb & 1);
        if (kb + 1 < nk) fetch((kb + 1) * kF64KC);
        const double *a_s = As + (size_t)buf * kF64KC * 128, *b_s = Bs + (size_t)buf * kF64KC * 128;
#pragma unroll
        for (int k = 0; k < kF64KC; ++k) {
            double a[8], b[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 x = *(const double2 *)(a_s + k * 128 + 2 * ty + 32 * i);
                const double2 y = *(const double2 *)(b_s + k * 128 + 2 * tx + 32 * i);
                a[2 * i] = x.x; a[2 * i + 1] = x.y;
                b[2 * i] = y.x; b[2 * i + 1] = y.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        // The other half was last read in the previous slice, before its barrier.
        if (kb + 1 < nk) stash(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t r = m0 + 2 * ty + 32 * (i >> 1) + (i & 1);
        if (r >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int64_t c = n0 + 2 * tx + 32 * (j >> 1) + (j & 1);
            if (c < N) C[r * ldc + c] = (float)acc[i][j];
        }
    }
}

// Workspace of the deferred-Q form: the recorded (c, s) of every round and
// the sorted positions, per slot.
__host__ inline size_t eig_dq_cs_bytes(int64_t pairs, int n, int max_sweeps) {
    return ((size_t)pairs * max_sweeps * n * n * sizeof(float2) + 255) & ~(size_t)255;
}
__host__ inline size_t eig_dq_bytes(int64_t pairs, int n, int max_sweeps) {
    return eig_dq_cs_bytes(pairs, n, max_sweeps) + (((size_t)pairs * n * 4 + 255) & ~(size_t)255);
}

template <int RPT, int CB, typename TG>
static int launch_eig_reg_dq(const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off, float *dmax,
                             int32_t *sweeps, int64_t pairs, int32_t max_sweeps, double tol, const double *live_floor,
                             unsigned char *dq_ws, cudaStream_t st) {
    constexpr int n = 32 * RPT;
    const size_t smem = eig_reg_smem_bytes(n, CB);
    float2 *cs = (float2 *)dq_ws;
    int *pos = (int *)(dq_ws + eig_dq_cs_bytes(pairs, n, max_sweeps));
    auto kern = eig_reg_kernel<RPT, CB, TG, true>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    kern<<<(unsigned)pairs, 32 * (n / CB), smem, st>>>(G, (__nv_bfloat16 *)Qt_hi, (__nv_bfloat16 *)Qt_lo,
                                                      (__nv_bfloat16 *)Qt_lo2, off, dmax, sweeps, max_sweeps, tol,
                                                      live_floor, cs, pos);
    if (cudaGetLastError() != cudaSuccess) return JB_ECUDA;
    const int64_t warps = pairs * n;
    q_apply_kernel<RPT><<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(cs, sweeps, pos, (__nv_bfloat16 *)Qt_hi,
                                                                     (__nv_bfloat16 *)Qt_lo, (__nv_bfloat16 *)Qt_lo2,
                                                                     (int)pairs, max_sweeps);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

template <int RPT, int CB, typename TG>
static int launch_eig_reg(const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off, float *dmax,
                          int32_t *sweeps, int64_t pairs, int32_t max_sweeps, double tol, const double *live_floor,
                          unsigned char *dq_ws, cudaStream_t st) {
    constexpr int n = 32 * RPT;
    const size_t smem = eig_reg_smem_bytes(n, CB);
    if (dq_ws)
        return launch_eig_reg_dq<RPT, CB, TG>(G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, max_sweeps, tol,
                                              live_floor, dq_ws, st);
    auto kern = eig_reg_kernel<RPT, CB, TG>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    kern<<<(unsigned)pairs, 32 * (n / CB), smem, st>>>(G, (__nv_bfloat16 *)Qt_hi, (__nv_bfloat16 *)Qt_lo,
                                                      (__nv_bfloat16 *)Qt_lo2, off, dmax, sweeps, max_sweeps, tol,
                                                      live_floor, nullptr, nullptr);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

template <typename TG>
static int dispatch_eig_reg(int n, int cb, const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off,
                            float *dmax, int32_t *sweeps, int64_t pairs, int32_t max_sweeps, double tol,
                            const double *live_floor, unsigned char *dq_ws, cudaStream_t st) {
#define JB_EIG_CASE(NN, RPT, CBV)                                                                               \
    if (n == NN && cb == CBV)                                                                                   \
        return launch_eig_reg<RPT, CBV, TG>(G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, max_sweeps, tol, \
                                            live_floor, dq_ws, st);
    JB_EIG_CASE(64, 2, 4)
    JB_EIG_CASE(64, 2, 8)
    JB_EIG_CASE(64, 2, 16)
    JB_EIG_CASE(128, 4, 4)
    // FP64 G with Q needs more registers than 512 threads have: 630 us two sweeps, with 256 threads 534
    if (sizeof(TG) == 8 && n == 128 && cb == 8 && !dq_ws) cb = 16;
    if constexpr (sizeof(TG) == 4) {
        JB_EIG_CASE(128, 4, 8)
    } else if (n == 128 && cb == 8) {
        return launch_eig_reg_dq<4, 8, TG>(G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, max_sweeps, tol,
                                           live_floor, dq_ws, st);
    }
    JB_EIG_CASE(128, 4, 16)
#undef JB_EIG_CASE
    return JB_EINVAL;
}

}  // namespace blk
}  // namespace jb

using namespace jb::blk;

extern "C" {

size_t jb_block_eig_workspace_bytes(int64_t pairs, int32_t n, int32_t max_sweeps) {
    if (pairs < 1 || n < 2 || max_sweeps < 1) return 0;
    return eig_dq_bytes(pairs, n, max_sweeps);
}

int jb_block_eig_ws(const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off, float *dmax,
                    int32_t *sweeps, int64_t pairs, int32_t n, int32_t max_sweeps, double tol,
                    const double *live_floor, int32_t variant, void *workspace, size_t workspace_bytes,
                    void *stream) {
    const bool dq = (variant & JB_EIG_DEFER_Q) != 0;
    variant &= ~JB_EIG_DEFER_Q;
    const int lay = variant & ~JB_EIG_FP32;
    if (!G || !Qt_hi || !Qt_lo || pairs < 1 || n < 2 || (n & 1) || max_sweeps < 1 ||
        !(lay == 0 || lay == 1 || lay == 4 || lay == 8 || lay == 16) || (variant & ~(JB_EIG_FP32 | 31)) ||
        ((variant & JB_EIG_FP32) && !((n == 64 || n == 128) && lay != 1)) ||
        (dq && !((n == 64 || n == 128) && lay != 1)))
        return JB_EINVAL;
    if (dq && (!workspace || workspace_bytes < eig_dq_bytes(pairs, n, max_sweeps))) return JB_EWORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const bool g32 = (variant & JB_EIG_FP32) != 0;
    const int layout = variant & ~JB_EIG_FP32;
    unsigned char *dq_ws = dq ? (unsigned char *)workspace : nullptr;
    if ((n == 64 || n == 128) && layout != 1) {
        const int cb = layout == 0 ? 8 : layout;
        return g32 ? dispatch_eig_reg<float>(n, cb, G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, max_sweeps,
                                             tol, live_floor, dq_ws, st)
                   : dispatch_eig_reg<double>(n, cb, G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, max_sweeps,
                                              tol, live_floor, dq_ws, st);
    }
    if (n > 256) return JB_ETOOBIG;                  // players are stored as bytes
    const size_t smem = eig_smem_bytes(n);
    if (smem > 227 * 1024) return JB_ETOOBIG;
    if (cudaFuncSetAttribute(eig_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    eig_kernel<<<(unsigned)pairs, kEigThreads, smem, st>>>(G, (__nv_bfloat16 *)Qt_hi, (__nv_bfloat16 *)Qt_lo,
                                                           (__nv_bfloat16 *)Qt_lo2, off, dmax, sweeps, n, max_sweeps,
                                                           tol, live_floor);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

int jb_block_eig_f64_ex(const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off, float *dmax,
                        int32_t *sweeps, int64_t pairs, int32_t n, int32_t max_sweeps, double tol,
                        const double *live_floor, int32_t variant, void *stream) {
    if (variant & JB_EIG_DEFER_Q) return JB_EWORKSPACE;  // the deferred-Q form needs jb_block_eig_ws
    return jb_block_eig_ws(G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, n, max_sweeps, tol, live_floor, variant,
                           nullptr, 0, stream);
}

int jb_block_eig_f64(const float *G, void *Qt_hi, void *Qt_lo, void *Qt_lo2, float *off, float *dmax,
                     int32_t *sweeps, int64_t pairs, int32_t n, int32_t max_sweeps, double tol, const double *live_floor,
                     void *stream) {
    return jb_block_eig_f64_ex(G, Qt_hi, Qt_lo, Qt_lo2, off, dmax, sweeps, pairs, n, max_sweeps, tol, live_floor, 0,
                               stream);
}

int jb_rows_scatter(const float *src, const int32_t *map, void *hi, void *lo, void *lo2, float *f32, int64_t rows,
                    int64_t L, void *stream) {
    if (!src || rows < 1 || L < 1 || (!hi && !f32)) return JB_EINVAL;
    dim3 grid((unsigned)((L + 255) / 256 > 64 ? 64 : (L + 255) / 256), (unsigned)(rows > 65535 ? 65535 : rows));
    scatter_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(src, map, (__nv_bfloat16 *)hi, (__nv_bfloat16 *)lo,
                                                           (__nv_bfloat16 *)lo2, f32, rows, L);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

int jb_rows_combine(const void *hi, const void *lo, const void *lo2, const int32_t *map, float *dst, int64_t rows,
                    int64_t L, void *stream) {
    if (!hi || !dst || rows < 1 || L < 1) return JB_EINVAL;
    dim3 grid((unsigned)((L + 255) / 256 > 64 ? 64 : (L + 255) / 256), (unsigned)(rows > 65535 ? 65535 : rows));
    combine_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)hi, (const __nv_bfloat16 *)lo,
                                                           (const __nv_bfloat16 *)lo2, map, dst, rows, L);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

int jb_block_finish(const float *Wt, const float *Vt, float *U, float *S, float *Vh, double *sig, int32_t *perm,
                    int64_t m, int64_t n, int32_t rank, int32_t e, int32_t cut_width, void *stream) {
    if (!Wt || !Vt || !S || !Vh || !U || !sig || !perm || m < 1 || n < 1 || rank < 1 || rank > n) return JB_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    norms_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(Wt, sig, n, m);
    rank_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(sig, perm, (int)n);
    const int64_t total = m * rank + (int64_t)rank * n + rank;
    int64_t blocks = (total + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    finish_kernel<<<(unsigned)blocks, 256, 0, st>>>(Wt, Vt, sig, perm, U, S, Vh, m, n, rank, e, cut_width);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

int jb_gemm_f64acc(const float *A, const float *B, float *C, int64_t M, int64_t N, int64_t K, int64_t lda,
                   int64_t ldb, int64_t ldc, void *stream) {
    if (!A || !B || !C || M < 1 || N < 1 || K < 1 || lda < K || ldb < K || ldc < N) return JB_EINVAL;
    if ((M + 127) / 128 > 65535) return JB_ETOOBIG;
    dim3 grid((unsigned)((N + 127) / 128), (unsigned)((M + 127) / 128));
    const bool vec = ((uintptr_t)A & 15) == 0 && ((uintptr_t)B & 15) == 0 && lda % 4 == 0 && ldb % 4 == 0 &&
                     K % 4 == 0;
    if (vec) {
        const int m_fast = N > M && (N + 127) / 128 <= 65535;
        if (m_fast) grid = dim3((unsigned)((M + 127) / 128), (unsigned)((N + 127) / 128));
        if (cudaFuncSetAttribute(gemm_f64acc_vec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kF64AccSmem) != cudaSuccess)
            return JB_ECUDA;
        gemm_f64acc_vec_kernel<<<grid, 256, kF64AccSmem, (cudaStream_t)stream>>>(A, B, C, M, N, K, lda, ldb, ldc,
                                                                                   m_fast);
    } else {
        gemm_f64acc_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(A, B, C, M, N, K, lda, ldb, ldc);
    }
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

}  // extern "C"
