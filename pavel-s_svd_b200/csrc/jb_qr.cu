// jb_qr.cu - batched Householder QR of tall matrices: the reference's
// primitives.qr (svdbench/standalone/primitives.py:74-89) with its
// reflector convention householder_vec (:41-59, LAPACK xLARFG: beta =
// -sign(alpha) ||x||, tau = (beta - alpha) / beta, v = x / (alpha - beta),
// v_0 = 1; a column with nothing below the diagonal is left alone) and Q by
// backward accumulation of the reflectors onto [I; 0].  It is the QR inside
// the reference's 'qr', 'tsqr' and projected ('randomized', 'subspace',
// 'block_krylov') solvers (solvers.py:71-96, 185-220, 245-248).
//
// All kernels compute in the input type, as the reference does.
//
// qr_panel_kernel: a cluster of 1 to 16 CTAs a matrix, each with a panel of rows
// in shared memory.  Per column j one reduction over the rows gives ||x||^2 and
// x^H y_c for all later columns at once (v = x / (alpha - beta), so v^H y_c =
// y_jc + x^H y_c / (alpha - beta)): one cluster barrier a column, every CTA
// pushing its sums into the others' shared memory before it.  Q = [I; 0] - V T
// V_1^H from the reflectors by rows, without further reductions: T^-1 =
// diag(1 / tau) + striu(V^H V), so T V_1^H is a triangular solve.  Bound by the
// latency of a column's step (about 1000 cycles).  B200: 2048 x 32 FP64 over 8
// CTAs 0.05 ms, 1.62 ms by one CTA through global memory; 256 x (256 x 16) FP32
// 0.02 ms, 0.07 ms.
//
// qr_kernel, cqr_kernel (matrices whose panels do not fit 16 SMs): one CTA per
// matrix (grid-stride over the batch).  The work area is the matrix (m x n,
// column-major: a warp walks a column with unit stride) whose lower part
// keeps the reflectors, and Q (m x n, column-major); in shared memory when
// both fit, else in a per-CTA slot of the workspace.  Per column j: the
// norm below the diagonal (one CTA reduction), the reflector, then one warp
// per remaining column applies I - tau v v^T.  Columns of Q left of j are
// zero in rows >= j during the backward accumulation, so only columns
// j..n-1 are updated (the reference's products with those zeros change
// nothing).
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <type_traits>
#include "jacobi_b200.h"

namespace jb {
namespace qr {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the CTA (partials in double); every thread gets it.  Two barriers.
template <typename T>
__device__ T block_sum(T v, double *red) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = (double)v;
    __syncthreads();
    double r = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += red[w];
    __syncthreads();
    return (T)r;
}

constexpr size_t kSmemLimit = 227 * 1024;

__device__ __forceinline__ float hyp(float a, float b) { return hypotf(a, b); }
__device__ __forceinline__ double hyp(double a, double b) { return hypot(a, b); }

__host__ __device__ inline size_t align16z(size_t x) { return (x + 15) & ~(size_t)15; }

// Shared memory: red (32 doubles) | tau (n) | [work area: 2 m n] when in_smem.
template <typename T>
__host__ __device__ inline size_t smem_bytes(int m, int n, bool in_smem) {
    return 32 * 8 + align16z((size_t)n * sizeof(T)) + (in_smem ? 2 * (size_t)m * n * sizeof(T) : 0);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) qr_kernel(const T *A, T *Qo, T *Ro, int64_t batch, int m, int n,
                                                      int in_smem, T *gws) {
    extern __shared__ __align__(16) unsigned char smem[];
    double *red = (double *)smem;
    T *tau = (T *)(smem + 32 * 8);
    const size_t mn = (size_t)m * n;
    T *Wk = in_smem ? (T *)(smem + 32 * 8 + align16z((size_t)n * sizeof(T))) : gws + (size_t)blockIdx.x * 2 * mn;
    T *Qk = Wk + mn;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int64_t z = blockIdx.x; z < batch; z += gridDim.x) {
        const T *a = A + z * (int64_t)mn;
        __syncthreads();
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int r = (int)(idx / n), c = (int)(idx - (size_t)r * n);
            Wk[(size_t)c * m + r] = a[idx];
        }
        __syncthreads();
        for (int j = 0; j < n; ++j) {
            T *x = Wk + (size_t)j * m;
            T part = T(0);
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) part += x[i] * x[i];
            const T xnorm = sqrt(block_sum(part, red));   // block_sum ends with a barrier
            const T alpha = x[j];
            const bool trivial = xnorm == T(0);
            const T beta = trivial ? alpha : (alpha < T(0) ? T(1) : T(-1)) * hyp(fabs(alpha), xnorm);
            const T denom = trivial ? T(1) : alpha - beta;
            const T t = trivial ? T(0) : (beta - alpha) / (beta != T(0) ? beta : T(1));
            __syncthreads();
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) x[i] = trivial ? T(0) : x[i] / denom;
            if (threadIdx.x == 0) { tau[j] = t; x[j] = beta; }
            __syncthreads();
            if (t != T(0)) {
                // columns j+1..n-1, rows j..m-1: y <- y - tau v (v^T y), v_j = 1
                for (int c = j + 1 + warp; c < n; c += nw) {
                    T *y = Wk + (size_t)c * m;
                    T w = T(0);
                    for (int i = j + lane; i < m; i += 32) w += (i == j ? T(1) : x[i]) * y[i];
                    w = warp_sum(w);
                    for (int i = j + lane; i < m; i += 32) y[i] -= t * (i == j ? T(1) : x[i]) * w;
                }
            }
            __syncthreads();
        }
        T *r = Ro + z * (int64_t)n * n;
        for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
            const int i = idx / n, c = idx - i * n;                   // R row-major, upper triangle
            r[idx] = i <= c ? Wk[(size_t)c * m + i] : T(0);
        }
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int c = (int)(idx / m), i = (int)(idx - (size_t)c * m);
            Qk[idx] = i == c ? T(1) : T(0);
        }
        __syncthreads();
        for (int j = n - 1; j >= 0; --j) {
            const T t = tau[j];
            if (t != T(0)) {
                const T *v = Wk + (size_t)j * m;
                for (int c = j + warp; c < n; c += nw) {
                    T *y = Qk + (size_t)c * m;
                    T w = T(0);
                    for (int i = j + lane; i < m; i += 32) w += (i == j ? T(1) : v[i]) * y[i];
                    w = warp_sum(w);
                    for (int i = j + lane; i < m; i += 32) y[i] -= t * (i == j ? T(1) : v[i]) * w;
                }
            }
            __syncthreads();
        }
        T *q = Qo + z * (int64_t)mn;
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int i = (int)(idx / n), c = (int)(idx - (size_t)i * n);   // Q row-major
            q[idx] = Qk[(size_t)c * m + i];
        }
    }
}

// Complex input (complex64 / complex128, interleaved re, im): the same
// algorithm with the reference's complex reflector (householder_vec for
// complex x: beta = -sign(Re alpha) hypot(|alpha|, ||x_2:||), real; the
// column is left alone only when nothing is below the diagonal AND alpha is
// real; tau = (beta - alpha) / beta and v = x / (alpha - beta) complex), the
// factorisation applying (I - conj(tau) v v^H) and Q accumulating
// (I - tau v v^H) as primitives.py:80-87 do.
template <typename R> struct Cx { R re, im; };
template <typename R> __device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {
    return Cx<R>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
template <typename R> __device__ __forceinline__ Cx<R> cmulc(Cx<R> a, Cx<R> b) {   // conj(a) b
    return Cx<R>{a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re};
}
template <typename R> __device__ __forceinline__ Cx<R> cdiv(Cx<R> a, Cx<R> b) {
    const R d = b.re * b.re + b.im * b.im;
    return Cx<R>{(a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d};
}

template <typename R>
__global__ void __launch_bounds__(kThreads) cqr_kernel(const Cx<R> *A, Cx<R> *Qo, Cx<R> *Ro, int64_t batch, int m,
                                                       int n, int in_smem, Cx<R> *gws) {
    using C = Cx<R>;
    extern __shared__ __align__(16) unsigned char smem[];
    double *red = (double *)smem;
    C *tau = (C *)(smem + 32 * 8);
    const size_t mn = (size_t)m * n;
    C *Wk = in_smem ? (C *)(smem + 32 * 8 + align16z((size_t)n * sizeof(C))) : gws + (size_t)blockIdx.x * 2 * mn;
    C *Qk = Wk + mn;
    const C zero{R(0), R(0)}, one{R(1), R(0)};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int64_t z = blockIdx.x; z < batch; z += gridDim.x) {
        const C *a = A + z * (int64_t)mn;
        __syncthreads();
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int r = (int)(idx / n), c = (int)(idx - (size_t)r * n);
            Wk[(size_t)c * m + r] = a[idx];
        }
        __syncthreads();
        for (int j = 0; j < n; ++j) {
            C *x = Wk + (size_t)j * m;
            R part = R(0);
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) part += x[i].re * x[i].re + x[i].im * x[i].im;
            const R xnorm = sqrt(block_sum(part, red));   // block_sum ends with a barrier
            const C alpha = x[j];
            const bool trivial = xnorm == R(0) && alpha.im == R(0);
            const R beta = trivial ? alpha.re
                                   : (alpha.re < R(0) ? R(1) : R(-1)) * hyp(hyp(alpha.re, alpha.im), xnorm);
            const C denom = trivial ? one : C{alpha.re - beta, alpha.im};
            const R bd = beta != R(0) ? beta : R(1);
            const C t = trivial ? zero : C{(beta - alpha.re) / bd, -alpha.im / bd};
            __syncthreads();
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) x[i] = trivial ? zero : cdiv(x[i], denom);
            if (threadIdx.x == 0) { tau[j] = t; x[j] = C{beta, R(0)}; }
            __syncthreads();
            if (t.re != R(0) || t.im != R(0)) {
                // columns j+1..n-1, rows j..m-1: y <- y - conj(tau) v (v^H y), v_j = 1
                const C tc{t.re, -t.im};
                for (int c = j + 1 + warp; c < n; c += nw) {
                    C *y = Wk + (size_t)c * m;
                    C w = zero;
                    for (int i = j + lane; i < m; i += 32) {
                        const C p = cmulc(i == j ? one : x[i], y[i]);
                        w.re += p.re; w.im += p.im;
                    }
                    w.re = warp_sum(w.re); w.im = warp_sum(w.im);
                    const C tw = cmul(tc, w);
                    for (int i = j + lane; i < m; i += 32) {
                        const C d = cmul(i == j ? one : x[i], tw);
                        y[i].re -= d.re; y[i].im -= d.im;
                    }
                }
            }
            __syncthreads();
        }
        C *r = Ro + z * (int64_t)n * n;
        for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
            const int i = idx / n, c = idx - i * n;
            r[idx] = i <= c ? Wk[(size_t)c * m + i] : zero;
        }
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int c = (int)(idx / m), i = (int)(idx - (size_t)c * m);
            Qk[idx] = i == c ? one : zero;
        }
        __syncthreads();
        for (int j = n - 1; j >= 0; --j) {
            const C t = tau[j];
            if (t.re != R(0) || t.im != R(0)) {
                const C *v = Wk + (size_t)j * m;
                for (int c = j + warp; c < n; c += nw) {
                    C *y = Qk + (size_t)c * m;
                    C w = zero;
                    for (int i = j + lane; i < m; i += 32) {
                        const C p = cmulc(i == j ? one : v[i], y[i]);
                        w.re += p.re; w.im += p.im;
                    }
                    w.re = warp_sum(w.re); w.im = warp_sum(w.im);
                    const C tw = cmul(t, w);
                    for (int i = j + lane; i < m; i += 32) {
                        const C d = cmul(i == j ? one : v[i], tw);
                        y[i].re -= d.re; y[i].im -= d.im;
                    }
                }
            }
            __syncthreads();
        }
        C *q = Qo + z * (int64_t)mn;
        for (size_t idx = threadIdx.x; idx < mn; idx += blockDim.x) {
            const int i = (int)(idx / n), c = (int)(idx - (size_t)i * n);
            q[idx] = Qk[(size_t)c * m + i];
        }
    }
}

// ---------------------------------------------------------------------------
// Panels over a cluster.
// ---------------------------------------------------------------------------
template <typename E> struct Num {   // real
    using R = E;
    static constexpr bool cx = false;
    __device__ static R low() { return sizeof(R) == 4 ? R(1e-30) : R(1e-280); }
    __device__ static R high() { return sizeof(R) == 4 ? R(1e38) : R(1e300); }
    __device__ static E make(R re, R) { return re; }
    __device__ static R re(E a) { return a; }
    __device__ static R im(E) { return R(0); }
};
template <typename T> struct Num<Cx<T>> {
    using R = T;
    static constexpr bool cx = true;
    __device__ static R low() { return Num<T>::low(); }
    __device__ static R high() { return Num<T>::high(); }
    __device__ static Cx<T> make(T re, T im) { return Cx<T>{re, im}; }
    __device__ static T re(Cx<T> a) { return a.re; }
    __device__ static T im(Cx<T> a) { return a.im; }
};
// acc + conj(a) b, acc - a b
__device__ __forceinline__ float fmac(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmac(double a, double b, double c) { return fma(a, b, c); }
template <typename T> __device__ __forceinline__ Cx<T> fmac(Cx<T> a, Cx<T> b, Cx<T> c) {
    return Cx<T>{fmac(a.re, b.re, fmac(a.im, b.im, c.re)), fmac(a.re, b.im, fmac(-a.im, b.re, c.im))};
}
__device__ __forceinline__ float fnma(float a, float b, float c) { return fmaf(-a, b, c); }
__device__ __forceinline__ double fnma(double a, double b, double c) { return fma(-a, b, c); }
template <typename T> __device__ __forceinline__ Cx<T> fnma(Cx<T> a, Cx<T> b, Cx<T> c) {
    return Cx<T>{fnma(a.re, b.re, fmac(a.im, b.im, c.re)), fnma(a.re, b.im, fnma(a.im, b.re, c.im))};
}
__device__ __forceinline__ float times(float a, float b) { return a * b; }
__device__ __forceinline__ double times(double a, double b) { return a * b; }
template <typename T> __device__ __forceinline__ Cx<T> times(Cx<T> a, Cx<T> b) { return cmul(a, b); }
__device__ __forceinline__ float plus(float a, float b) { return a + b; }
__device__ __forceinline__ double plus(double a, double b) { return a + b; }
template <typename T> __device__ __forceinline__ Cx<T> plus(Cx<T> a, Cx<T> b) { return Cx<T>{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ float conj_of(float a) { return a; }
__device__ __forceinline__ double conj_of(double a) { return a; }
template <typename T> __device__ __forceinline__ Cx<T> conj_of(Cx<T> a) { return Cx<T>{a.re, -a.im}; }
__device__ __forceinline__ float wsum(float a) { return warp_sum(a); }
__device__ __forceinline__ double wsum(double a) { return warp_sum(a); }
template <typename T> __device__ __forceinline__ Cx<T> wsum(Cx<T> a) { return Cx<T>{warp_sum(a.re), warp_sum(a.im)}; }

template <int CS> __device__ __forceinline__ void team_barrier() {
    if constexpr (CS == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int CS> __device__ __forceinline__ unsigned team_rank() {
    unsigned r = 0;
    if constexpr (CS > 1) asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
// *ptr of CTA `rank` in the cluster = v
template <int CS, typename E> __device__ __forceinline__ void push(E *ptr, unsigned rank, E v) {
    if constexpr (CS == 1) {
        *ptr = v;
    } else {
        unsigned a;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(ptr)), "r"(rank));
        if constexpr (sizeof(E) == 4) {
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
        } else if constexpr (!Num<E>::cx) {
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
        } else if constexpr (sizeof(E) == 8) {
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.re), "f"(v.im) : "memory");
        } else {
            asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.re), "d"(v.im) : "memory");
        }
    }
}

// f with the number of columns a warp takes at once (1, 2 or 4) for `left` columns.
template <typename F> __device__ __forceinline__ void panel_wide(int left, F f) {
    if (left > kThreads / 16) f(std::integral_constant<int, 4>());
    else if (left > kThreads / 32) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 1>());
}

// Shared memory: sums 2 x CS x n | row 2 x n | tau n | X n x n | panel n x (rows + 1)
template <typename E>
__host__ __device__ inline size_t panel_smem(int rows, int n, int cs) {
    return ((size_t)2 * cs * n + 2 * n + n + (size_t)n * n + (size_t)n * (rows + 1)) * sizeof(E);
}

template <typename E, int CS>
__global__ void __launch_bounds__(kThreads) qr_panel_kernel(const E *A, E *Qo, E *Ro, int64_t batch, int m, int n,
                                                            int rows) {
    using N = Num<E>;
    using R = typename N::R;
    extern __shared__ __align__(16) unsigned char smem[];
    E *sums = (E *)smem;                     // [parity][rank][column]
    E *rowj = sums + 2 * CS * n;             // [parity][column]
    E *tau = rowj + 2 * n;
    E *X = tau + n;                          // strict lower: (V^H V)^T, upper: M = T V_1^H
    E *P = X + n * n;                        // column c at c * ld
    const int ld = rows + 1;                 // the transposing load hits every bank
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NW = kThreads / 32;
    const unsigned rank = team_rank<CS>();
    const int row0 = rank * rows, mine = min(max(m - row0, 0), rows);
    const E zero = N::make(R(0), R(0)), one = N::make(R(1), R(0));
    for (int64_t z = blockIdx.x / CS; z < batch; z += gridDim.x / CS) {
        const E *a = A + z * (int64_t)m * n + (int64_t)row0 * n;
        for (int idx = threadIdx.x; idx < rows * n; idx += kThreads) {
            const int i = idx / n, c = idx - i * n;
            P[c * ld + i] = i < mine ? a[idx] : zero;
        }
        __syncthreads();
        for (int j = 0; j < n; ++j) {
            const int par = j & 1;
            const E *x = P + j * ld;
            // x^H y_c over this panel's rows below j, to every CTA; row j from its owner
            const int lo = rank == 0 ? j + 1 : 0;
            panel_wide(n - j, [&](auto width) {
                constexpr int U = decltype(width)::value;
                for (int c0 = j + warp; c0 < n; c0 += U * NW) {
                    const E *y[U];
                    E w[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        y[u] = P + min(c0 + u * NW, n - 1) * ld;
                        w[u] = zero;
                    }
                    for (int i = lo + lane; i < rows; i += 32) {
                        const E v = x[i];
#pragma unroll
                        for (int u = 0; u < U; ++u) w[u] = fmac(v, y[u][i], w[u]);
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) w[u] = wsum(w[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int c = c0 + u * NW;
                        if (c >= n) continue;
                        if (lane < CS) push<CS>(sums + (par * CS + rank) * n + c, lane, w[u]);
                        if (rank == 0 && lane < CS) push<CS>(rowj + par * n + c, lane, y[u][j]);
                    }
                }
            });
            team_barrier<CS>();
            E s = zero;
#pragma unroll
            for (int q = 0; q < CS; ++q) s = plus(s, sums[(par * CS + q) * n + j]);
            const R x2 = N::re(s);
            const E alpha = rowj[par * n + j];
            const bool trivial = x2 == R(0) && N::im(alpha) == R(0);
            // ||(alpha, x)||: by squares unless alpha's leave the range
            const R a2 = N::re(alpha) * N::re(alpha) + N::im(alpha) * N::im(alpha), b2 = a2 + x2;
            R norm;
            if (b2 > Num<E>::low() && b2 < Num<E>::high()) norm = sqrt(b2);
            else norm = hyp(N::cx ? hyp(N::re(alpha), N::im(alpha)) : fabs(N::re(alpha)), sqrt(x2));
            const R beta = trivial ? N::re(alpha) : (N::re(alpha) < R(0) ? norm : -norm);
            const R bd = beta != R(0) ? beta : R(1);
            const E t = trivial ? zero : N::make((beta - N::re(alpha)) / bd, -N::im(alpha) / bd);
            // 1 / (alpha - beta)
            const R dr = N::re(alpha) - beta, di = N::im(alpha), dn = dr * dr + di * di;
            const E inv = trivial ? zero : (N::cx ? N::make(dr / dn, -di / dn) : N::make(R(1) / dr, R(0)));
            if (!trivial) {
                panel_wide(n - j - 1, [&](auto width) {
                    constexpr int U = decltype(width)::value;
                    for (int c0 = j + 1 + warp; c0 < n; c0 += U * NW) {
                        E *y[U];
                        E f[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int c = min(c0 + u * NW, n - 1);
                            y[u] = P + c * ld;
                            E w = zero;
#pragma unroll
                            for (int q = 0; q < CS; ++q) w = plus(w, sums[(par * CS + q) * n + c]);
                            // v^H y_c = y_jc + conj(inv) x^H y_c; y <- y - conj(tau) v (v^H y)
                            w = times(conj_of(t), plus(rowj[par * n + c], times(conj_of(inv), w)));
                            f[u] = times(inv, w);
                            if (rank == 0 && lane == u && c0 + u * NW < n) y[u][j] = fnma(one, w, y[u][j]);
                        }
                        for (int i = lo + lane; i < rows; i += 32) {
                            const E v = x[i];
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                if (c0 + u * NW < n) y[u][i] = fnma(v, f[u], y[u][i]);
                        }
                    }
                });
            }
            __syncthreads();   // all dot products and updates with x are done
            if (warp == (j & (NW - 1))) {
                E *v = P + j * ld;
                for (int i = lo + lane; i < rows; i += 32) v[i] = times(v[i], inv);
                if (rank == 0 && lane == 0) v[j] = N::make(beta, R(0));
                if (lane == 0) tau[j] = t;
            }
        }
        __syncthreads();
        if (rank == 0) {
            // R out, then the unit lower triangle in its place
            E *r = Ro + z * (int64_t)n * n;
            for (int idx = threadIdx.x; idx < n * n; idx += kThreads) {
                const int i = idx / n, c = idx - i * n;
                r[idx] = i <= c ? P[c * ld + i] : zero;
                if (i <= c) P[c * ld + i] = i == c ? one : zero;
            }
        }
        // (V^H V)(i, c), i < c, of this panel at X(c, i): 4 x 4 tiles a warp, lanes over rows
        __syncthreads();
        const int nt = (n + 3) >> 2;
        for (int b = warp; b < nt * (nt + 1) / 2; b += NW) {
            int bc = 0, bi = b;
            while (bi > bc) { bi -= bc + 1; ++bc; }     // bi <= bc
            E acc[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = zero;
            for (int i = lane; i < rows; i += 32) {
                E xa[4], ya[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    xa[u] = P[min(4 * bi + u, n - 1) * ld + i];
                    ya[u] = P[min(4 * bc + u, n - 1) * ld + i];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] = fmac(xa[u], ya[v], acc[u][v]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const E w = wsum(acc[u][v]);
                    const int i = 4 * bi + u, c = 4 * bc + v;
                    if (lane == 0 && i < c && c < n) X[c * n + i] = w;
                }
        }
        if constexpr (CS > 1) {
            team_barrier<CS>();
            // sum of the panels' parts, in place of the upper triangle (X(i, c))
            for (int idx = threadIdx.x; idx < n * n; idx += kThreads) {
                const int c = idx / n, i = idx - c * n;
                if (i >= c) continue;
                E w = zero;
#pragma unroll
                for (int q = 0; q < CS; ++q) {
                    unsigned ad;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;"
                        : "=r"(ad) : "r"((unsigned)__cvta_generic_to_shared(X + c * n + i)), "r"((unsigned)q));
                    E v;
                    if constexpr (sizeof(E) == 4) {
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ad) : "memory");
                    } else if constexpr (!N::cx) {
                        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ad) : "memory");
                    } else if constexpr (sizeof(E) == 8) {
                        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.re), "=f"(v.im) : "r"(ad) : "memory");
                    } else {
                        asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.re), "=d"(v.im) : "r"(ad) : "memory");
                    }
                    w = plus(w, v);
                }
                X[i * n + c] = w;
            }
            team_barrier<CS>();   // everyone has read the parts
            for (int idx = threadIdx.x; idx < n * n; idx += kThreads) {
                const int c = idx / n, i = idx - c * n;
                if (i < c) X[c * n + i] = X[i * n + c];
            }
            team_barrier<CS>();   // ... and has its upper triangle free
        }
        // V_1^H's columns to every CTA: row c of V_1 is in panel 0
        if (rank == 0)
            for (int idx = threadIdx.x; idx < n * n * CS; idx += kThreads) {
                const int q = idx / (n * n), k = idx - q * n * n, c = k / n, i = k - c * n;
                if (i <= c) push<CS>(X + i * n + c, q, conj_of(P[i * ld + c]));
            }
        team_barrier<CS>();
        // M_i = tau_i (b_i - sum_(k > i) (V^H V)_ik M_k), column c by one thread
        for (int c = threadIdx.x; c < n; c += kThreads)
            for (int i = c; i >= 0; --i) {
                E w = X[i * n + c];
                for (int k = i + 1; k <= c; ++k) w = fnma(X[k * n + i], X[k * n + c], w);
                X[i * n + c] = times(tau[i], w);
            }
        __syncthreads();
        // Q = [I; 0] - V M
        E *q = Qo + z * (int64_t)m * n + (int64_t)row0 * n;
        const int rt = (mine + 3) >> 2;
        for (int b = threadIdx.x; b < rt * nt; b += kThreads) {
            const int bc = b % nt, bi = b / nt;
            E acc[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = zero;
            const int kmax = min(4 * bc + 3, n - 1);
            for (int k = 0; k <= kmax; ++k) {
                E xa[4], ya[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    xa[u] = P[k * ld + min(bi + u * rt, rows - 1)];
                    const int c = min(4 * bc + u, n - 1);
                    ya[u] = k <= c ? X[k * n + c] : zero;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] = fnma(xa[u], ya[v], acc[u][v]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int i = bi + u * rt, c = 4 * bc + v;
                    if (i < mine && c < n) q[(int64_t)i * n + c] = plus(acc[u][v], row0 + i == c ? one : zero);
                }
        }
        team_barrier<CS>();   // nobody pushes into a CTA still at this matrix
    }
}

static int sm_count_of_device() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))
        return 0;
    return sms;
}

template <typename T>
static bool fits_smem(int m, int n) {
    return smem_bytes<T>(m, n, true) <= kSmemLimit;
}

template <typename T, typename K>
static int launch(K kern, const T *A, T *Q, T *R, int64_t batch, int m, int n, void *workspace, size_t ws_bytes,
                  cudaStream_t st) {
    const bool in_smem = fits_smem<T>(m, n);
    const size_t smem = smem_bytes<T>(m, n, in_smem);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess) return JB_ECUDA;
    const int sms = sm_count_of_device();
    if (sms <= 0 || per_sm < 1) return JB_ECUDA;
    int64_t grid = (int64_t)sms * per_sm;
    if (grid > batch) grid = batch;
    T *gws = nullptr;
    if (!in_smem) {
        const size_t per_cta = 2 * (size_t)m * n * sizeof(T);
        const int64_t fit = (int64_t)(ws_bytes / per_cta);
        if (!workspace || fit < 1) return JB_EWORKSPACE;
        if (grid > fit) grid = fit;
        gws = (T *)workspace;
    }
    kern<<<(unsigned)grid, kThreads, smem, st>>>(A, Q, R, batch, m, n, in_smem ? 1 : 0, gws);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

// Panels: the cluster size for a shape and batch, 0 when a matrix does not fit 16
// SMs (8 is the portable limit; 16 only for what needs it).  The fewest CTAs whose panels fit (96 KB, so that two share an SM),
// then more while the batch leaves SMs idle and a panel keeps 64 rows and n.
template <typename E>
static int panel_cluster(int m, int n, int64_t batch, int sms) {
    auto rows_of = [&](int cs) { return ((m + cs - 1) / cs + 31) & ~31; };
    int cs = 1;
    while (cs < 8 && panel_smem<E>(rows_of(cs), n, cs) > 96 * 1024) cs *= 2;
    if (panel_smem<E>(rows_of(cs), n, cs) > kSmemLimit) cs = 16;
    while (cs < 8 && batch * cs * 2 <= sms && rows_of(2 * cs) >= 64) cs *= 2;
    while (cs > 1 && rows_of(cs) < n) cs /= 2;
    return panel_smem<E>(rows_of(cs), n, cs) <= kSmemLimit ? cs : 0;
}

template <typename T>
static size_t workspace_bytes(int m, int n, int64_t batch) {
    if (fits_smem<T>(m, n)) return 0;
    int sms = sm_count_of_device();
    if (sms <= 0) sms = 148;
    if (panel_cluster<T>(m, n, batch, sms)) return 0;
    const int64_t grid = batch < (int64_t)sms * 2 ? batch : (int64_t)sms * 2;
    return (size_t)grid * 2 * (size_t)m * n * sizeof(T);
}

template <typename E, int CS>
static int launch_panel(const E *A, E *Q, E *R, int64_t batch, int m, int n, cudaStream_t st) {
    auto kern = qr_panel_kernel<E, CS>;
    const int rows = ((m + CS - 1) / CS + 31) & ~31;
    const size_t smem = panel_smem<E>(rows, n, CS);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return JB_ECUDA;
    if (CS > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return JB_ECUDA;
    const int64_t teams = batch < (1 << 16) ? batch : (1 << 16);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(teams * CS));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CS > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, A, Q, R, batch, m, n, rows) == cudaSuccess ? JB_OK : JB_ECUDA;
}

template <typename T, typename K>
static int entry(K kern, const T *A, T *Q, T *R, int64_t batch, int32_t m, int32_t n, void *workspace,
                 size_t ws_bytes, void *stream) {
    if (!A || !Q || !R || batch < 0 || n < 1 || m < n) return JB_EINVAL;
    if ((int64_t)m * n > ((int64_t)1 << 31)) return JB_ETOOBIG;
    if (batch == 0) return JB_OK;
    const int sms = sm_count_of_device();
    if (sms <= 0) return JB_ECUDA;
    switch (panel_cluster<T>(m, n, batch, sms)) {
        case 1: return launch_panel<T, 1>(A, Q, R, batch, m, n, (cudaStream_t)stream);
        case 2: return launch_panel<T, 2>(A, Q, R, batch, m, n, (cudaStream_t)stream);
        case 4: return launch_panel<T, 4>(A, Q, R, batch, m, n, (cudaStream_t)stream);
        case 8: return launch_panel<T, 8>(A, Q, R, batch, m, n, (cudaStream_t)stream);
        case 16: return launch_panel<T, 16>(A, Q, R, batch, m, n, (cudaStream_t)stream);
    }
    return launch<T>(kern, A, Q, R, batch, m, n, workspace, ws_bytes, (cudaStream_t)stream);
}

}  // namespace qr
}  // namespace jb

extern "C" {

size_t jb_qr_workspace_bytes(int32_t m, int32_t n, int64_t batch, int32_t elem) {
    if (n < 1 || m < n || batch < 0) return 0;
    if (elem == 16) return jb::qr::workspace_bytes<jb::qr::Cx<double>>(m, n, batch);
    return elem == 8 ? jb::qr::workspace_bytes<double>(m, n, batch) : jb::qr::workspace_bytes<float>(m, n, batch);
}

int jb_qr_f32(const float *A, float *Q, float *R, int64_t batch, int32_t m, int32_t n, void *workspace,
              size_t workspace_bytes, void *stream) {
    return jb::qr::entry<float>(jb::qr::qr_kernel<float>, A, Q, R, batch, m, n, workspace, workspace_bytes, stream);
}

int jb_qr_f64(const double *A, double *Q, double *R, int64_t batch, int32_t m, int32_t n, void *workspace,
              size_t workspace_bytes, void *stream) {
    return jb::qr::entry<double>(jb::qr::qr_kernel<double>, A, Q, R, batch, m, n, workspace, workspace_bytes,
                                 stream);
}

int jb_qr_c64(const void *A, void *Q, void *R, int64_t batch, int32_t m, int32_t n, void *workspace,
              size_t workspace_bytes, void *stream) {
    using E = jb::qr::Cx<float>;
    return jb::qr::entry<E>(jb::qr::cqr_kernel<float>, (const E *)A, (E *)Q, (E *)R, batch, m, n, workspace,
                            workspace_bytes, stream);
}

int jb_qr_c128(const void *A, void *Q, void *R, int64_t batch, int32_t m, int32_t n, void *workspace,
               size_t workspace_bytes, void *stream) {
    using E = jb::qr::Cx<double>;
    return jb::qr::entry<E>(jb::qr::cqr_kernel<double>, (const E *)A, (E *)Q, (E *)R, batch, m, n, workspace,
                            workspace_bytes, stream);
}

}  // extern "C"
