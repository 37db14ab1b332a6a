// jb_mixed.cuh - the mixed-precision solve of float32 matrices up to 256 x 128
// (tall view): a preconditioned FP32 Jacobi, then an FP64 refinement made of
// matrix products.
//
//   factor_kernel (128 threads a matrix)
//     G = A^T A in FP64 (mma f64), pivoted Cholesky P^T G P = L L^T in FP64;
//     L rounded to FP32.
//   precondition_kernel (64 threads a matrix)
//     one-sided FP32 Jacobi of L.  A = Q L^T P^T, so the left singular vectors
//     of L are the right singular vectors of A: the rotated and normalised
//     columns are V, and no V is accumulated.  L is n x n and
//     its columns start out graded (Veselic and Hari; Drmac and Veselic), so
//     a sweep moves n instead of m + n rows a column and fewer sweeps are
//     needed (128 x 64 with singular values over three decades: 7 instead of
//     13).
//   refine_kernel (256 threads a matrix; refine_large_kernel above 128 x 64, a
//   cluster of CTAs)
//     repeat: E = V^T V - I, W = A V from the exact input, H = W^T W (FP64);
//     done when every pair ratio |h_pq| / sqrt(h_pp h_qq) is <= tol -- the
//     reference's convergence test on the current W (primitives.py:334-339,
//     352-353) -- and V is orthogonal to 1e-8; else V <- V (I + N), N = K -
//     E / 2 with K the skew matrix of all Jacobi angles of H at once
//     (primitives.py:340-346), which leaves the square of the errors (the
//     refinement of Ogita and Aishima).  Usually one correction.
//
// Measured (B200, 8192 matrices n ~ U[8,64], m ~ U[n,2n]; ms a batch): factor
// 0.33, precondition 0.86, refine 1.01, against 4.55 + 3.03 of the register
// kernels' FP32 and FP64 phases from V = I; 4096 x 128 x 64 over three decades
// 0.38 + 1.00 + 1.04 against 12.9; one 256 x 128 over four decades 0.14 + 0.41 +
// 0.15 against 4.1 + 2.3.  U is also closer to LAPACK's (1.4e-7 against
// 1.4e-6: all pairs are corrected, not only those above tol).
//
// A matrix that this does not suit -- numerically rank-deficient, full bases
// wanted, no convergence within its passes -- is marked kPending and solved by
// the launches that follow (rb32_kernel_t, rb64_kernel).
#pragma once
#include "jb_device.cuh"

namespace jb {

constexpr int kPending = -1;   // status: left to the register kernels
constexpr int kHanded = -2;    // status: FP32 sweeps done by rb32, FP64 phase due
constexpr int kFacT = 128, kPreT = 64, kRefT = 256, kRefNarrowT = 128;
// A pivot below kPivotCut times the largest diagonal of G (a singular value
// ratio of about 3e-6) is left to the register kernels: FP64 rounding of G
// no longer resolves it well enough for a start.
constexpr double kPivotCut = 1e-11;
constexpr int kRefPasses = 6;
constexpr double kRefOrth = 1e-8;

__host__ __device__ inline int round8(int x) { return (x + 7) & ~7; }
// Smallest 4 * odd >= x: with it as a leading dimension in doubles (or the
// row stride in floats) the 8 x 4 lane pattern of the f64 mma fragments hits
// every bank once; 8 * odd does so for floats along the other index.
__host__ __device__ inline int ld4odd(int x) { const int q = (x + 3) >> 2; return 4 * (q | 1); }
__host__ __device__ inline int ld8odd(int x) { const int q = (x + 7) >> 3; return 8 * (q | 1); }

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// The tall view of A as FP32 in shared memory, zero-padded to m8 x n8:
// element (i, k) at i * sr + k * sk, the fast index as in the input, so that
// reads of the input are coalesced and stores conflict-free.
struct Stage { int sr, sk; };
__host__ __device__ inline Stage stage_of(bool wide, int m8, int n8) {
    return wide ? Stage{1, ld8odd(m8)} : Stage{ld4odd(n8), 1};
}
__host__ __device__ inline size_t stage_floats(int m8, int n8) {
    const size_t a = (size_t)m8 * ld4odd(n8), b = (size_t)n8 * ld8odd(m8);
    return a > b ? a : b;
}
// Asynchronous copies (global to shared, zeros past the input): all of a
// thread's loads are in flight at once.  Rows in quads when the input allows.
__device__ __forceinline__ void cp_async4(float *dst, const float *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
template <int THREADS>
__device__ __forceinline__ void stage_input(const float *A, int rows, int cols, int rows8, int cols8, int ld,
                                            float *As) {
    // input rows x cols (row-major), padded with zeros; the thread's column
    // and row advance by a fixed step
    const bool quads = (cols & 3) == 0 && ((uintptr_t)A & 15) == 0;
    const int width = quads ? cols8 >> 2 : cols8;
    const int step_r = THREADS / width, step_c = THREADS - step_r * width;
    int r = threadIdx.x / width, c = threadIdx.x - r * width;
    while (r < rows8) {
        if (quads) {
            const bool in = r < rows && 4 * c < cols;
            cp_async16(As + r * ld + 4 * c, in ? A + (size_t)r * cols + 4 * c : A, in);
        } else {
            const bool in = r < rows && c < cols;
            cp_async4(As + r * ld + c, in ? A + (size_t)r * cols + c : A, in);
        }
        r += step_r;
        c += step_c;
        if (c >= width) { c -= width; ++r; }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void stage_tall(const float *A, const jb_matrix_desc &d, int m8, int n8, Stage st, float *As,
                                           int threads) {
    if (threads == 128) {
        if (d.m < d.n) stage_input<128>(A, d.m, d.n, n8, m8, st.sk, As);
        else stage_input<128>(A, d.m, d.n, m8, n8, st.sr, As);
    } else {
        if (d.m < d.n) stage_input<256>(A, d.m, d.n, n8, m8, st.sk, As);
        else stage_input<256>(A, d.m, d.n, m8, n8, st.sr, As);
    }
}

// ---------------------------------------------------------------------------
// FP32 Jacobi with GL = 8 lanes a block pair (16 above 64 columns): lane gl of a group owns R rows of
// the 2B columns of its two blocks.  Compared with a whole warp a pair
// (jb_regblock.cuh) a step's fixed cost -- the reductions, the rotation
// parameters, the broadcasts -- is shared by four pairs of blocks a warp:
// about 8 instead of 39 instructions a column pair at 64 rows.  Eight
// groups hold all columns, so a matrix needs two warps.  Issue-bound (62 % of
// the issue slots at 16 warps an SM, registers the limit); plain instead of
// scaled rotations, unrolled intra steps and the factor in the same kernel (12
// warps an SM) took 1.62 ms for factor and sweeps on the uneven batch, 1.19 now.
// ---------------------------------------------------------------------------
// The columns are kept scaled, w = scale * (the tile's column): a rotation is
// then x - a y, y + b x with both columns' scales multiplied by c (Gentleman's
// square-root-free rotation), half the arithmetic of the plain form.  Scales
// start at 1 each sweep and shrink by at most sqrt(2) a rotation.
template <int GL, int B, int R>
struct GTile {
    float w[2 * B][R];
    // of the lane's pair (x_i, y_i), i = the lane's position in the group / (GL / B):
    float nx, ny;   // squared norms
    float dx, dy;   // scales
};

template <int R>
__device__ __forceinline__ float gdot(const float (&x)[R], const float (&y)[R]) {
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int r = 0; r < R; r += 2) fma2(a0, a1, x[r], x[r + 1], y[r], y[r + 1]);
    return a0 + a1;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The rotation of rot_params<float> as its tangent t (with the sign of apq)
// and c, on approximate reciprocals without denormal handling: the squared
// norms here are above kPivotCut of the largest, which is about 1.  Returns
// bit 0: active, bit 2: ratio > the exit ratio.  Inactive: t = 0, c = 1.
__device__ __forceinline__ int gparams(float app, float aqq, float apq, float tol2, float ex2, float &t, float &c) {
    const float apq2 = apq * apq, prod = app * aqq;
    const bool active = apq2 > tol2 * prod && fminf(app, aqq) > 0.f;
    const float d = aqq - app;
    const float h = fmaf(d, d, 4.f * apq2);
    const float tt = 2.f * apq * rcp_ftz(fabsf(d) + h * rsqrt_ftz(h));
    t = active ? (d < 0.f ? -tt : tt) : 0.f;
    const float x = fmaf(t, t, 1.f);
    const float c0 = rsqrt_ftz(x);
    c = c0 * fmaf(-0.5f * x, c0 * c0, 1.5f);
    return active ? 1 | (apq2 > ex2 * prod ? 4 : 0) : 0;
}
// x <- x - a y, y <- y + b x
template <int R>
__device__ __forceinline__ void grot(float (&x)[R], float (&y)[R], float a, float b) {
    const float2 na = make_float2(-a, -a), pb = make_float2(b, b);
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        const float2 u = make_float2(x[r], x[r + 1]), v = make_float2(y[r], y[r + 1]);
        const float2 u2 = __ffma2_rn(na, v, u), v2 = __ffma2_rn(pb, u, v);
        x[r] = u2.x; x[r + 1] = u2.y;
        y[r] = v2.x; y[r + 1] = v2.y;
    }
}

// B pairs of the group's columns: INTRA pairs columns inside each block, with
// scales 1 and exact norms, and applies c; otherwise x_i with y_i, norms and
// scales kept by the lanes of pair i.
template <bool INTRA, int GL, int B, int R>
__device__ __forceinline__ void gstep(GTile<GL, B, R> &t, float tol2, float ex2, int &fl, int lane) {
    constexpr int LB = Log2<B>::value, LG = Log2<GL>::value;
    float pc[B];
#pragma unroll
    for (int i = 0; i < B; ++i) pc[i] = gdot(t.w[pair_p<INTRA, B>(i)], t.w[pair_q<INTRA, B>(i)]);
    lanes_reduce_scatter<GL>(pc, lane);
    float tn, c;
    if constexpr (INTRA) {
        float pa[B], pb[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int p = pair_p<INTRA, B>(i), q = pair_q<INTRA, B>(i);
            pa[i] = gdot(t.w[p], t.w[p]);
            pb[i] = gdot(t.w[q], t.w[q]);
        }
        lanes_reduce_scatter<GL>(pa, lane);
        lanes_reduce_scatter<GL>(pb, lane);
        fl |= gparams(pa[0], pb[0], pc[0], tol2, ex2, tn, c);
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int src = (lane & ~(GL - 1)) | (i << (LG - LB));
            const float ti = __shfl_sync(FULL, tn, src), ci = __shfl_sync(FULL, c, src);
            const int p = pair_p<INTRA, B>(i), q = pair_q<INTRA, B>(i);
            grot(t.w[p], t.w[q], ti, ti);
#pragma unroll
            for (int r = 0; r < R; ++r) { t.w[p][r] *= ci; t.w[q][r] *= ci; }
        }
    } else {
        const float apq = pc[0] * (t.dx * t.dy);
        const int f = gparams(t.nx, t.ny, apq, tol2, ex2, tn, c);
        fl |= f;
        if (!__any_sync(FULL, f != 0)) return;
        const float sh = tn * apq;
        const float a = tn * (t.dy * rcp_ftz(t.dx)), b = tn * (t.dx * rcp_ftz(t.dy));
        t.nx -= sh;
        t.ny += sh;
        t.dx *= c;
        t.dy *= c;
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int src = (lane & ~(GL - 1)) | (i << (LG - LB));
            grot(t.w[i], t.w[B + i], __shfl_sync(FULL, a, src), __shfl_sync(FULL, b, src));
        }
    }
}

template <int GL, int B, int R>
__device__ __forceinline__ void gcircle(GTile<GL, B, R> &t) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int o = half * B;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float last = t.w[o + B - 1][r];
#pragma unroll
            for (int i = B - 1; i >= 2; --i) t.w[o + i][r] = t.w[o + i - 1][r];
            if (B > 1) t.w[o + 1][r] = last;
        }
    }
}
template <int GL, int B, int R>
__device__ __forceinline__ void gshift_y(GTile<GL, B, R> &t, int lane) {
    const int from = (lane & ~(GL - 1)) | ((lane + GL / B) & (GL - 1));
    t.ny = __shfl_sync(FULL, t.ny, from);
    t.dy = __shfl_sync(FULL, t.dy, from);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float f = t.w[B][r];
#pragma unroll
        for (int i = 0; i < B - 1; ++i) t.w[B + i][r] = t.w[B + i + 1][r];
        t.w[2 * B - 1][r] = f;
    }
}

// Row of register r of lane gl: chunks of 4 (then 2) consecutive rows, chunk
// by chunk over the lanes, so that a group's vector access to a column in the
// exchange area is one run of 128 (64) bytes.
template <int GL, int R>
__device__ __forceinline__ int grow(int r, int gl) {
    return r < (R & ~3) ? (r >> 2) * 4 * GL + gl * 4 + (r & 3) : (R & ~3) * GL + gl * (R & 3) + (r - (R & ~3));
}
template <int GL, int B, int R, bool STORE>
__device__ __forceinline__ void gtile_x(GTile<GL, B, R> &t, float *xw, int X, int Y, int gl) {
#pragma unroll
    for (int c = 0; c < 2 * B; ++c) {
        float *col = xw + (c < B ? X * B + c : Y * B + (c - B)) * (GL * R);
#pragma unroll
        for (int k = 0; k < R / 4; ++k) {
            float4 *p = (float4 *)(col + k * 4 * GL) + gl;
            if (STORE) *p = make_float4(t.w[c][4 * k], t.w[c][4 * k + 1], t.w[c][4 * k + 2], t.w[c][4 * k + 3]);
            else {
                const float4 v = *p;
                t.w[c][4 * k] = v.x; t.w[c][4 * k + 1] = v.y; t.w[c][4 * k + 2] = v.z; t.w[c][4 * k + 3] = v.w;
            }
        }
        if (R & 2) {
            float2 *p = (float2 *)(col + (R & ~3) * GL) + gl;
            if (STORE) *p = make_float2(t.w[c][R - 2], t.w[c][R - 1]);
            else {
                const float2 v = *p;
                t.w[c][R - 2] = v.x; t.w[c][R - 1] = v.y;
            }
        }
    }
}

// Sweeps over L (x, n x n, column-major) until no pair ratio of a sweep
// exceeds exit_ratio; then the normalised columns take L's place.  xb: the
// exchange area.  Returns the sweeps, or max_sweeps + 1.
template <int GL, int B, int R>
__device__ int precondition_sweeps(float *xb, int n, float exit_ratio, int max_sweeps, float *x) {
    constexpr int LB = Log2<B>::value, LG = Log2<GL>::value;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & (GL - 1);
    const int group = threadIdx.x / GL;
    const int nb = 2 * ((n + 2 * B - 1) / (2 * B));
    const bool act = group < nb / 2, wact = warp * (32 / GL) < nb / 2;
    const int li = gl >> (LG - LB), base = lane & ~(GL - 1);
    float2 *xn = (float2 *)(xb + nb * B * GL * R);
    GTile<GL, B, R> t;
    int X = act ? group : 0, Y = act ? nb - 1 - group : 0;
#pragma unroll
    for (int c = 0; c < 2 * B; ++c) {
        const int col = c < B ? X * B + c : Y * B + (c - B);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = grow<GL, R>(r, gl);
            t.w[c][r] = act && col < n && row < n ? x[col * n + row] : 0.f;
        }
    }
    const float tol = 10.f * Lim<float>::eps();
    const float tol2 = tol * tol, ex2 = exit_ratio * exit_ratio;
    int sweep = 1;
    for (; sweep <= max_sweeps; ++sweep) {
        int fl = 0;
        if (wact) {
            if (sweep > 1) {   // back to scales 1
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const float sx = __shfl_sync(FULL, t.dx, base | (i << (LG - LB)));
                    const float sy = __shfl_sync(FULL, t.dy, base | (i << (LG - LB)));
#pragma unroll
                    for (int r = 0; r < R; ++r) { t.w[i][r] *= sx; t.w[B + i][r] *= sy; }
                }
            }
            if constexpr (B > 1) {
#pragma unroll 1
                for (int j = 0; j < B - 1; ++j) {
                    gstep<true>(t, tol2, ex2, fl, lane);
                    gcircle(t);
                }
            }
            float nrm[2 * B];   // exact norms: column j's on lanes j * GL / 2B ...
#pragma unroll
            for (int c = 0; c < 2 * B; ++c) nrm[c] = gdot(t.w[c], t.w[c]);
            lanes_reduce_scatter<GL>(nrm, lane);
            t.nx = __shfl_sync(FULL, nrm[0], base | (li << (LG - 1 - LB)));
            t.ny = __shfl_sync(FULL, nrm[0], base | ((B + li) << (LG - 1 - LB)));
            t.dx = t.dy = 1.f;
        }
#pragma unroll 1
        for (int br = 0; br < nb - 1; ++br) {
            if (br > 0 || sweep > 1) {
                if (act) {
                    gtile_x<GL, B, R, true>(t, xb, X, Y, gl);
                    if ((gl & (GL / B - 1)) == 0) {
                        xn[X * B + li] = make_float2(t.nx, t.dx);
                        xn[Y * B + li] = make_float2(t.ny, t.dy);
                    }
                }
                __syncthreads();
                if (act) {
                    if (X > 0) X = X == 1 ? nb - 1 : X - 1;
                    Y = Y == 1 ? nb - 1 : Y - 1;
                    gtile_x<GL, B, R, false>(t, xb, X, Y, gl);
                    const float2 u = xn[X * B + li], v = xn[Y * B + li];
                    t.nx = u.x; t.dx = u.y;
                    t.ny = v.x; t.dy = v.y;
                }
            }
            if (wact) {
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    gstep<false>(t, tol2, ex2, fl, lane);
                    gshift_y(t, lane);
                }
            }
        }
        if (!__syncthreads_or(fl & 4)) break;
    }
    if (sweep > max_sweeps) return sweep;
    if (wact) {
        float nrm[2 * B];
#pragma unroll
        for (int c = 0; c < 2 * B; ++c) nrm[c] = gdot(t.w[c], t.w[c]);
        lanes_reduce_scatter<GL>(nrm, lane);
#pragma unroll
        for (int c = 0; c < 2 * B; ++c) {
            const float inv = 1.f / sqrtf(__shfl_sync(FULL, nrm[0], base | (c << (LG - 1 - LB))));
            const int col = c < B ? X * B + c : Y * B + (c - B);
            if (act && col < n) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int row = grow<GL, R>(r, gl);
                    if (row < n) x[col * n + row] = t.w[c][r] * inv;
                }
            }
        }
    }
    return sweep;
}

__host__ __device__ inline size_t pre_smem(int nt) {
    const size_t cols = nt > 32 ? (nt + 7) / 8 * 8 : nt > 16 ? (nt + 3) / 4 * 4 : (nt + 1) / 2 * 2;
    const size_t rows = nt > 96 ? 128 : nt > 64 ? 96 : nt > 48 ? 64 : nt > 32 ? 48 : nt > 16 ? 32 : 16;
    return cols * rows * 4 + cols * 8;
}

// THREADS 64 up to 64 columns, 256 up to 128 (which also takes the narrower
// matrices of such a batch).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kPreT ? 8 : 1) precondition_kernel(Params p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_idx;
    float *xb = (float *)smem;
    const float exit_ratio = p.exit_ratio == 0.f ? kMixedExitRatio
                                                 : (p.exit_ratio < 0.f ? 10.f * Lim<float>::eps() : p.exit_ratio);
    for (;;) {
        int64_t idx;
        next_ticket(p.counter, s_idx, idx);
        if (idx >= p.count) break;
        const int64_t mat = p.order ? (int64_t)p.order[idx] : idx;
        const jb_matrix_desc d = desc_of(p, mat);
        if (p.status[mat] != JB_ST_OK) continue;
        const int nt = d.m > d.n ? d.n : d.m, most = p.max_sweeps32;
        float *x = p.x32 + d.x_off;
        int ns = 0;
        if (THREADS > kPreT && nt > 64) {
            if constexpr (THREADS > kPreT) {
                if (nt > 96) ns = precondition_sweeps<16, 4, 8>(xb, nt, exit_ratio, most, x);
                else ns = precondition_sweeps<16, 4, 6>(xb, nt, exit_ratio, most, x);
            }
        } else if (nt > 48) ns = precondition_sweeps<8, 4, 8>(xb, nt, exit_ratio, most, x);
        else if (nt > 32) ns = precondition_sweeps<8, 4, 6>(xb, nt, exit_ratio, most, x);
        else if (nt > 16) ns = precondition_sweeps<8, 2, 4>(xb, nt, exit_ratio, most, x);
        else ns = precondition_sweeps<8, 1, 2>(xb, nt, exit_ratio, most, x);
        if (threadIdx.x == 0) {
            p.sweeps[mat] = ns;
            if (ns > most) {
                p.status[mat] = kPending;
                atomicAdd(p.n_pending, 1);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// The factor L.
// ---------------------------------------------------------------------------
// Pivoted Cholesky of G (n x n, both triangles, ld), thread i = row i, by one
// warp (n <= 32), two or four.  Step k takes the largest remaining diagonal, row
// p at column position q; every thread swaps columns k and q of its own row,
// so that columns 0 .. k - 1 of a row hold L's and both factors of a dot
// product are runs of shared memory (ld = 2 mod 4: conflict-free 16-byte reads,
// row p a broadcast).  At the end G(i, k) is column k of L (0 in rows chosen
// before).  The pivot is found on FP32 keys that carry the row (redux); one
// barrier a step.  scl brings the largest diagonal to about 1, rscl is its
// square root.  False when a pivot is <= cut (scaled).
template <int WARPS>
__device__ __forceinline__ bool pivoted_cholesky(double *G, int ld, int n, double cut, double scl, double rscl,
                                                 double2 *sd, int *spos, unsigned *skey) {
    constexpr unsigned M = WARPS == 4 ? 127u : 63u;   // the key's bits for the row
    const int i = threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool row = i < n;
    double *gi = G + min(i, n - 1) * ld;
    double d = row ? gi[i] : 0.0;
    bool taken = !row;
    int pos = i;
    for (int k = 0; k < n; ++k) {
        const float df = (float)(d * scl);
        const unsigned key = taken ? 0u : ((__float_as_uint(fmaxf(df, 0.f)) & ~M) | (M - i)) + (M + 1u);
        unsigned kw = __reduce_max_sync(FULL, key);
        // 1 / sqrt(d): FP32 estimate, one Newton step (1e-14)
        const double r0 = (double)rsqrt_ftz(df);
        const double rs = r0 * fma(-0.5 * (d * scl), r0 * r0, 1.5) * rscl;
        if (!taken) {
            sd[i] = make_double2(d, rs);
            spos[i] = pos;
        }
        if (WARPS > 1) {
            if (lane == 0) skey[WARPS * (k & 1) + warp] = kw;
            asm volatile("bar.sync 1, %0;" ::"n"(32 * WARPS) : "memory");
            const unsigned *ks = skey + WARPS * (k & 1);
#pragma unroll
            for (int w = 0; w < WARPS; ++w) kw = max(kw, ks[w]);
        } else {
            __syncwarp();
        }
        const int p = (int)(M - (kw & M));
        const double2 dr = sd[p];
        const int q = spos[p];
        if (!(dr.x * scl > cut)) return false;
        const double *gp = G + p * ld;
        const double g = gi[q], gk = gi[k];
        double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
        int j = 0;
#pragma unroll 2
        for (; j + 8 <= k; j += 8) {
#pragma unroll
            for (int t = 0; t < 8; t += 4) {
                const double2 a = *(const double2 *)(gi + j + t), b = *(const double2 *)(gp + j + t);
                const double2 e = *(const double2 *)(gi + j + t + 2), f = *(const double2 *)(gp + j + t + 2);
                v0 = fma(a.x, b.x, v0);
                v1 = fma(a.y, b.y, v1);
                v2 = fma(e.x, f.x, v2);
                v3 = fma(e.y, f.y, v3);
            }
        }
#pragma unroll 1
        for (; j + 2 <= k; j += 2) {
            const double2 a = *(const double2 *)(gi + j), b = *(const double2 *)(gp + j);
            v0 = fma(a.x, b.x, v0);
            v1 = fma(a.y, b.y, v1);
        }
        if (j < k) v2 = fma(gi[j], gp[j], v2);
        const double l = taken ? 0.0 : (i == p ? dr.x : g - ((v0 + v1) + (v2 + v3))) * dr.y;
        if (row) {
            gi[q] = gk;
            gi[k] = l;
        }
        if (i == p) taken = true;
        else if (pos == k) pos = q;
        d = fma(-l, l, d);
    }
    return true;
}

// Shared memory: spos (N ints), sd (N double2), skey (8), sex (8), then G (n8
// rows of n8 + 2 doubles) and the staged input in one place; N = 64 or 128 columns.
template <int N> struct FacHead { static constexpr size_t bytes = N * 4 + N * 16 + 8 * 4 + 8 * 4; };
template <int N>
__host__ __device__ inline size_t fac_smem(int mt, int nt) {
    const int m8 = round8(mt), n8 = round8(nt);
    const size_t g = (size_t)n8 * (n8 + 2) * 8, a = stage_floats(m8, n8) * 4;
    return FacHead<N>::bytes + (g > a ? g : a);
}

// Lower 16 x 16 blocks of G over WARPS warps, at most JOBS a warp; all sums stay
// in registers until the staged input is no longer needed.
template <int JOBS, int WARPS>
__device__ __forceinline__ void gram_tiles(const float *As, Stage st, int m8, int nt8, double *G, int ld) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    double acc[JOBS][2][2][2];
    int tr[JOBS], tc[JOBS];
    bool own[JOBS];
#pragma unroll
    for (int j = 0; j < JOBS; ++j) {
        int g = 0, job = warp + WARPS * j;   // block row g has g + 1 blocks
        while (job > g) { job -= g + 1; ++g; }
        tr[j] = 2 * g;
        tc[j] = 2 * job;
        own[j] = tr[j] < nt8;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) acc[j][a][b][0] = acc[j][a][b][1] = 0.0;
    }
    const int last = nt8 - 1;
    const float *a0 = As + lk * st.sr + lr * st.sk;
#pragma unroll 2
    for (int k0 = 0; k0 < m8; k0 += 4, a0 += 4 * st.sr) {
#pragma unroll
        for (int j = 0; j < JOBS; ++j) {
            if (!own[j]) continue;
            double fa[2], fb[2];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                fa[a] = (double)a0[min(tr[j] + a, last) * 8 * st.sk];
                fb[a] = (double)a0[min(tc[j] + a, last) * 8 * st.sk];
            }
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) dmma(acc[j][a][b], fa[a], fb[b]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < JOBS; ++j)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (tr[j] + a >= nt8 || tc[j] + b > tr[j] + a) continue;
                const int r = (tr[j] + a) * 8 + lr, c = (tc[j] + b) * 8 + 2 * lk;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    G[(size_t)r * ld + c + e] = acc[j][a][b][e];
                    if (tc[j] + b < tr[j] + a) G[(size_t)(c + e) * ld + r] = acc[j][a][b][e];
                }
            }
    __syncthreads();
}

// THREADS 128 up to 128 x 64, 256 up to 256 x 128.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kFacT ? 6 : 1) factor_kernel(Params p) {
    constexpr bool BIG = THREADS != kFacT;
    constexpr int N = BIG ? 128 : 64;
    extern __shared__ __align__(16) unsigned char smem[];
    int *spos = (int *)smem;
    double2 *sd = (double2 *)(smem + N * 4);
    unsigned *skey = (unsigned *)(smem + N * 4 + N * 16);
    int *sex = (int *)(skey + 8);
    double *G = (double *)(smem + FacHead<N>::bytes);
    for (int64_t idx = blockIdx.x; idx < p.count; idx += gridDim.x) {
        const int64_t mat = p.order ? (int64_t)p.order[idx] : idx;
        const jb_matrix_desc d = desc_of(p, mat);
        int st = JB_ST_OK;
        const int mt = d.m > d.n ? d.m : d.n, nt = d.m > d.n ? d.n : d.m;
        if (!rdesc_fits(d, kB32, 4, p, true, BIG ? kMaxRL : kMaxR, BIG ? kMaxRVL : kMaxRV)) {
            st = JB_ST_BAD_DESC;
        } else if ((d.flags & JB_FULL_MATRICES) && mt > nt) {
            st = kPending;
        } else {
            const int m8 = round8(mt), n8 = round8(nt), ld = n8 + 2;
            const Stage sg = stage_of(d.m < d.n, m8, n8);
            float *As = (float *)G;
            stage_tall((const float *)p.A + d.a_off, d, m8, n8, sg, As, THREADS);
            __syncthreads();
            if (BIG) gram_tiles<5, THREADS / 32>(As, sg, m8, n8 >> 3, G, ld);
            else if (nt > 32) gram_tiles<3, THREADS / 32>(As, sg, m8, n8 >> 3, G, ld);
            else gram_tiles<1, THREADS / 32>(As, sg, m8, n8 >> 3, G, ld);
            // a diagonal of G is not finite exactly when the input is not
            const double gd = threadIdx.x < nt ? G[(size_t)threadIdx.x * ld + threadIdx.x] : 0.0;
            const int ex = __reduce_max_sync(FULL, (__double2hiint(fabs(gd)) >> 20) & 0x7ff);
            if ((threadIdx.x & 31) == 0) sex[threadIdx.x >> 5] = ex;
            const bool bad = __syncthreads_or(!isfinite(gd));
            int em = sex[0];   // the warps that hold rows
#pragma unroll
            for (int w = 1; w < N / 32; ++w) em = max(em, sex[w]);
            if (bad) {
                st = JB_ST_NONFINITE_IN;
            } else if (em < 32) {
                st = kPending;   // zero, or the squares near the bottom of FP64's range
            } else {
                // even power of two that brings the largest diagonal into [1, 4)
                const int half = (em - 1023) >> 1;
                const double scl = __hiloint2double((1023 - 2 * half) << 20, 0);
                const double rscl = __hiloint2double((1023 - half) << 20, 0);
                bool ok = true;
                if (BIG && nt > 64) {
                    if (threadIdx.x < 128) ok = pivoted_cholesky<4>(G, ld, nt, kPivotCut, scl, rscl, sd, spos, skey);
                } else if (nt > 32) {
                    if (threadIdx.x < 64) ok = pivoted_cholesky<2>(G, ld, nt, kPivotCut, scl, rscl, sd, spos, skey);
                } else {
                    if (threadIdx.x < 32) ok = pivoted_cholesky<1>(G, ld, nt, kPivotCut, scl, rscl, sd, spos, skey);
                }
                if (__syncthreads_or(!ok)) {
                    st = kPending;
                } else {
                    float *x = p.x32 + d.x_off;
                    for (int c = threadIdx.x >> 5; c < nt; c += THREADS / 32)
                        for (int i = threadIdx.x & 31; i < nt; i += 32)
                            x[c * nt + i] = (float)(G[i * ld + c] * rscl);
                }
            }
        }
        if (threadIdx.x == 0) {
            p.status[mat] = st;
            p.sweeps[mat] = 0;
            if (st == kPending) atomicAdd(p.n_pending, 1);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// FP64 refinement.  Eight warps a matrix; V (n8 x ldv) and W (n8 x ldw,
// column-major, FP64) in shared memory, the staged input and N in W's place
// while W is not needed: 102 KB at 128 x 64, two matrices an SM.  The floor is
// the f64 mma pipe, 4 n^3 + 6 m n^2 flop for the usual one correction and its
// check (0.30 ms of the uneven batch's 1.01); barriers between the products
// and the shared-memory latency of their operands take the rest.
// ---------------------------------------------------------------------------
struct RefGeo {
    int m8, n8, ldv, ldw;
};
__host__ __device__ inline RefGeo ref_geo(int mt, int nt) {
    RefGeo r;
    r.m8 = round8(mt);
    r.n8 = round8(nt);
    r.ldv = ld4odd(r.n8);
    r.ldw = ld4odd(r.m8);
    return r;
}
__host__ __device__ inline size_t ref_smem(int mt, int nt) {
    const RefGeo r = ref_geo(mt, nt);
    size_t w = (size_t)r.n8 * r.ldw * 8;
    const size_t a = stage_floats(r.m8, r.n8) * 4;
    if (a > w) w = a;
    return (size_t)r.n8 * r.ldv * 8 + w + (size_t)64 * 8 * 3 + 64 * 4;
}

// C (mt8 x nt8 tiles, column-major) = (ADD ? C : 0) + X Y over k8, in blocks
// of 16 rows and NB column tiles a warp, S blocks a warp at most.  X(i, k) at
// x[i * sr + k * sk], Y(k, j) at y[j * ldy + k].  C is written once every
// warp is done reading: it may take X's or Y's place.  Rows and columns of a
// block past the end repeat the last tile; their results are not stored.
template <int NB, int S, int NW, bool ADD, typename TX>
__device__ __forceinline__ void ref_mul(const TX *x, int sr, int sk, const double *y, int ldy, double *C, int ldc,
                                        int k8, int mt8, int nt8) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    const int bm = (mt8 + 1) >> 1, blocks = bm * ((nt8 + NB - 1) / NB);
    double acc[S][2][NB][2];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int blk = warp + NW * s;
#pragma unroll
        for (int b = 0; b < NB; ++b)
            acc[s][0][b][0] = acc[s][0][b][1] = acc[s][1][b][0] = acc[s][1][b][1] = 0.0;
        if (blk < blocks) {
            const int tr = 2 * (blk % bm), tc = NB * (blk / bm);
            const TX *xa = x + (tr * 8 + lr) * sr + lk * sk;
            const TX *xb = x + (min(tr + 1, mt8 - 1) * 8 + lr) * sr + lk * sk;
            const double *yb[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) yb[b] = y + (min(tc + b, nt8 - 1) * 8 + lr) * ldy + lk;
#pragma unroll 2
            for (int k0 = 0; k0 < k8; k0 += 4) {
                const double fa = (double)xa[k0 * sk], fb = (double)xb[k0 * sk];
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const double f = yb[b][k0];
                    dmma(acc[s][0][b], fa, f);
                    dmma(acc[s][1][b], fb, f);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int blk = warp + NW * s;
        if (blk < blocks) {
            const int tr = 2 * (blk % bm), tc = NB * (blk / bm);
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    if (tr + a < mt8 && tc + b < nt8) {
                        double *w = C + ((tc + b) * 8 + 2 * lk) * ldc + (tr + a) * 8 + lr;
                        w[0] = acc[s][a][b][0] + (ADD ? w[0] : 0.0);
                        w[ldc] = acc[s][a][b][1] + (ADD ? w[ldc] : 0.0);
                    }
        }
    }
}
// W = A V with A staged in W's place, and V <- V + V N, with the block width
// (3 or 4 column tiles) that leaves the fewest idle.
template <int NB, int NW>
__device__ __forceinline__ void ref_w(const float *As, Stage st, const double *V, int ldv, double *W, int ldw, int mt8,
                                      int nt8) {
    ref_mul<NB, 2, NW, false>(As, st.sr, st.sk, V, ldv, W, ldw, 8 * nt8, mt8, nt8);
}
template <int NB, int NW>
__device__ __forceinline__ void ref_v(double *V, int ldv, const double *Nm, int nt8) {
    ref_mul<NB, 1, NW, true>(V, 1, ldv, Nm, ldv, V, ldv, 8 * nt8, nt8, nt8);
}
__device__ __forceinline__ bool ref_three(int nt8) { return nt8 == 3 || nt8 == 5 || nt8 == 6; }

// Lower 16 x 8 blocks of X^T X (X column-major, ld, rows8 rows): three jobs a warp at most.
__device__ __forceinline__ void job_place(int job, int &tr, int &tc) {
    // block row g (16 rows) has 2 g + 2 column tiles
    int g = 0;
    while (job >= 2 * g + 2) { job -= 2 * g + 2; ++g; }
    tr = 2 * g;
    tc = job;
}
__device__ __forceinline__ void ref_gram(const double *X, int ld, int rows8, int tr, int tc, int nt8,
                                         double (&acc)[2][2]) {
    const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    const double *x0 = X + (size_t)(tr * 8 + lr) * ld + lk;
    const double *x1 = X + (size_t)((tr + 1 < nt8 ? tr + 1 : tr) * 8 + lr) * ld + lk;
    const double *y = X + (size_t)(tc * 8 + lr) * ld + lk;
    acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0.0;
#pragma unroll 4
    for (int k = 0; k < rows8; k += 4) {
        const double b = y[k];
        dmma(acc[0], x0[k], b);
        dmma(acc[1], x1[k], b);
    }
}

// tan of the Jacobi angle of (d = h_qq - h_pp, h_pq) in FP32 from
// exponent-scaled inputs: its relative error of 1e-7 is one of the
// correction only.
__device__ __forceinline__ double ref_angle(double d, double a) {
    const double a2 = 2.0 * a;
    const int ex = (__double2hiint(fmax(fabs(d), fabs(a2))) >> 20) & 0x7ff;
    if (ex == 0) return 0.0;
    const double scl = __hiloint2double((2046 - ex) << 20, 0);
    const float df = fabsf((float)(d * scl)), af = (float)(a2 * scl);
    const float hf = fmaf(df, df, af * af);
    const float t = __fdividef(af, df + hf * rsqrtf(hf));
    return d < 0.0 ? -(double)t : (double)t;
}

// THREADS 256 (two matrices an SM at 128 x 64), or 128 for matrices of at most 32
// columns (four or more an SM).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) refine_kernel(Params p) {
    constexpr int NW = THREADS / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_idx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    for (;;) {
        int64_t idx;
        next_ticket(p.counter2, s_idx, idx);
        if (idx >= p.count) break;
        const int mat = p.order ? p.order[idx] : (int)idx;
        if (p.status[mat] != JB_ST_OK) continue;
        int mt, nt;
        bool wide;
        {
            const jb_matrix_desc d = desc_of(p, mat);
            if (!class_takes(d, p.cls)) continue;   // the other size class's launch refines it
            wide = d.m < d.n;
            mt = wide ? d.n : d.m;
            nt = wide ? d.m : d.n;
        }
        const RefGeo g = ref_geo(mt, nt);
        const int ldv = g.ldv, ldw = g.ldw, nt8 = g.n8 >> 3, mt8 = g.m8 >> 3;
        double *dh = (double *)smem, *de = dh + 64, *sig = de + 64;   // diagonals of H and E; sigma
        int *perm = (int *)(sig + 64);
        double *V = (double *)(perm + 64);
        double *W = V + (size_t)g.n8 * ldv;
        double *Nm = W;                       // n8 x ldv
        float *As = (float *)W;
        const Stage sg = stage_of(wide, g.m8, g.n8);
        {
            const float *x = p.x32 + desc_of(p, mat).x_off;
            for (int c = warp; c < g.n8; c += NW)
                for (int i = lane; i < g.n8; i += 32)
                    V[c * ldv + i] = (c < nt && i < nt) ? (double)x[c * nt + i] : 0.0;
        }
        const int nb16 = (nt8 + 1) >> 1, jobs = nb16 * (nb16 + 1);
        const int most = p.max_sweeps < kRefPasses ? p.max_sweeps : kRefPasses;
        int pass = 1;
        bool done = false;
        for (; pass <= most; ++pass) {
            {
                const jb_matrix_desc d = desc_of(p, mat);
                stage_tall((const float *)p.A + d.a_off, d, g.m8, g.n8, sg, As, THREADS);
            }
            __syncthreads();
            if (ref_three(nt8)) ref_w<3, NW>(As, sg, V, ldv, W, ldw, mt8, nt8);
            else ref_w<4, NW>(As, sg, V, ldv, W, ldw, mt8, nt8);
            __syncthreads();
            double h[3][2][2], e[3][2][2];
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int job = warp + NW * s;
                if (job >= jobs) continue;
                int tr, tc;
                job_place(job, tr, tc);
                if (tc >= nt8) continue;
                ref_gram(W, ldw, g.m8, tr, tc, nt8, h[s]);
                ref_gram(V, ldv, g.n8, tr, tc, nt8, e[s]);
#pragma unroll
                for (int a = 0; a < 2; ++a)
                    if (tr + a == tc) {   // diagonal tile: lanes with column 2 lk or 2 lk + 1 == row lr
                        const int r = tc * 8 + lr;
                        if ((lr >> 1) == lk) {
                            const double ee = (lr & 1 ? e[s][a][1] : e[s][a][0]) - 1.0;
                            dh[r] = lr & 1 ? h[s][a][1] : h[s][a][0];
                            de[r] = r < nt ? ee : 0.0;
                        }
                    }
            }
            __syncthreads();
            const double tol = p.tol > 0 ? (double)(float)p.tol : (double)(10.0f * Lim<float>::eps());
            const double tol2 = tol * tol;
            int need = 0;
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int job = warp + NW * s;
                if (job >= jobs) continue;
                int tr, tc;
                job_place(job, tr, tc);
                if (tc >= nt8) continue;
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int r = (tr + a) * 8 + lr, c = tc * 8 + 2 * lk + u;
                        if (r < nt && c < r) {
                            if (!(h[s][a][u] * h[s][a][u] <= tol2 * dh[r] * dh[c])) need = 1;
                            if (!(fabs(e[s][a][u]) <= kRefOrth)) need = 1;
                        } else if (r < nt && c == r) {
                            if (!(fabs(de[r]) <= kRefOrth)) need = 1;
                        }
                    }
            }
            if (!__syncthreads_or(need)) { done = true; break; }
            if (pass == most) break;
            // N = K - E / 2, column-major in W's place
            int wild = 0;
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int job = warp + NW * s;
                if (job >= jobs) continue;
                int tr, tc;
                job_place(job, tr, tc);
                if (tc >= nt8) continue;
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int r = (tr + a) * 8 + lr, c = tc * 8 + 2 * lk + u;
                        if (tr + a >= nt8 || c > r) continue;
                        if (r >= nt) {
                            Nm[r * ldv + c] = 0.0;
                            Nm[c * ldv + r] = 0.0;
                        } else if (c == r) {
                            Nm[c * ldv + r] = -0.5 * de[r];
                        } else {
                            // rotation of columns c < r of W: h without what E explains of it
                            const double ee = e[s][a][u];
                            const double off = h[s][a][u] - 0.5 * ee * (dh[r] + dh[c]);
                            const double k = ref_angle(dh[r] * (1.0 - de[r]) - dh[c] * (1.0 - de[c]), off);
                            if (!(fabs(k) <= 0.25 && fabs(ee) <= 0.1)) wild = 1;
                            Nm[r * ldv + c] = k - 0.5 * ee;
                            Nm[c * ldv + r] = -k - 0.5 * ee;
                        }
                    }
            }
            if (__syncthreads_or(wild)) { pass = most; break; }
            // second-order term on the diagonal: -sum_i K_ij^2 / 2 (an isolated
            // close pair has an angle far above all others)
            for (int j = warp; j < nt; j += NW) {
                double sum = 0.0;
                for (int i = lane; i < nt; i += 32) {
                    const double k = 0.5 * (Nm[j * ldv + i] - Nm[i * ldv + j]);
                    sum = fma(k, k, sum);
                }
                sum = warp_sum(sum);
                if (lane == 0) Nm[j * ldv + j] -= 0.5 * sum;
            }
            __syncthreads();
            if (ref_three(nt8)) ref_v<3, NW>(V, ldv, Nm, nt8);
            else ref_v<4, NW>(V, ldv, Nm, nt8);
        }
        // sigma, the stable descending order and the cut (primitives.py:356-366)
        int st = JB_ST_OK;
        if (done) {
            if (threadIdx.x < nt) sig[threadIdx.x] = sqrt(dh[threadIdx.x]);
            __syncthreads();
            int below = 0;
            if (threadIdx.x < 4 * nt) {   // four threads count a column's rank
                const int j = threadIdx.x >> 2;
                const double sj = sig[j];
                int rnk = 0;
                double smax = 0.0;
                for (int i = threadIdx.x & 3; i < nt; i += 4) {
                    const double si = sig[i];
                    rnk += (si > sj) || (si == sj && i < j);
                    smax = fmax(smax, si);
                }
                const unsigned quad = 0xfu << (lane & ~3);
                rnk += __shfl_xor_sync(quad, rnk, 1);
                rnk += __shfl_xor_sync(quad, rnk, 2);
                smax = fmax(smax, __shfl_xor_sync(quad, smax, 1));
                smax = fmax(smax, __shfl_xor_sync(quad, smax, 2));
                const int npref = nt + (nt & 1);
                below = !(sj > Lim<double>::eps() * (mt > npref ? mt : npref) * smax);
                if ((threadIdx.x & 3) == 0) perm[rnk] = j;
            }
            if (__syncthreads_or(below)) done = false;   // columns to complete: not here
        }
        if (!done) {
            st = kPending;
        } else {
            const jb_matrix_desc d = desc_of(p, mat);
            float *U = p.U ? (float *)p.U + d.u_off : nullptr;
            float *Vh = p.Vh ? (float *)p.Vh + d.v_off : nullptr;
            float *S = (float *)p.S + d.s_off;
            int bad = 0;
            if (threadIdx.x < d.rank) {
                const float o = (float)sig[perm[threadIdx.x]];
                if (!isfinite(o)) bad = 1;
                S[threadIdx.x] = o;
            }
            if (!(d.flags & JB_VALUES_ONLY)) {
                if (threadIdx.x < nt) dh[threadIdx.x] = 1.0 / sig[threadIdx.x];
                __syncthreads();
                // left factor X (rows x rank, row-major): 8 ranks x 4 rows a warp and step
                const double *X = wide ? V : W;
                const int ldl = wide ? ldv : ldw, rows = wide ? nt : mt;
                const int r8 = (d.rank + 7) >> 3;
                for (int blk = warp; blk < ((rows + 3) >> 2) * r8; blk += NW) {
                    const int r = (blk % r8) * 8 + (lane & 7), i = (blk / r8) * 4 + (lane >> 3);
                    if (r < d.rank && i < rows) {
                        const int c = perm[r];
                        const float o = (float)(wide ? X[c * ldl + i] : X[c * ldl + i] * dh[c]);
                        if (!isfinite(o)) bad = 1;
                        U[(size_t)i * d.rank + r] = o;
                    }
                }
                const double *Y = wide ? W : V;
                const int ldr = wide ? ldw : ldv, cols = wide ? mt : nt;
                for (int r = warp; r < d.rank; r += NW) {
                    const int c = perm[r];
                    const double f = wide ? dh[c] : 1.0;
                    for (int i = lane; i < cols; i += 32) {
                        const float o = (float)(Y[c * ldr + i] * f);
                        if (!isfinite(o)) bad = 1;
                        Vh[(size_t)r * cols + i] = o;
                    }
                }
            }
            if (__syncthreads_or(bad)) st = JB_ST_NONFINITE_OUT;
        }
        if (threadIdx.x == 0) {
            p.status[mat] = st;
            if (st == kPending) atomicAdd(p.n_pending, 1);
            else p.sweeps[mat] += pass;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// FP64 refinement above 128 x 64 (up to 256 x 128): the same passes by a cluster
// of CTAs a matrix, as W (266 KB) does not fit one SM.  Every CTA keeps all of
// V and 32 rows of W in shared memory.  Per pass: W rows = A rows V; the CTA's
// part of H = W^T W to the workspace (16 x 16 blocks in mma layout); each CTA
// then sums its share of the blocks over the parts, forms E and N there, and
// writes N into the shared memory of the CTAs that own its columns; these
// update their columns of V and write them into every CTA's copy.  Four
// cluster barriers a pass.  One matrix uses 8 SMs instead of one: 256 x 128 in
// 0.145 ms, against 2.31 ms for gram64_kernel.
// ---------------------------------------------------------------------------
constexpr int kLgRows = 32, kLgN = 128;

struct LgGeo {
    int n8, ldv, nb16, gpc;   // padded width, its ld, 16-column groups, groups a CTA
};
__host__ __device__ inline LgGeo lg_geo(int nt, int cs) {
    LgGeo g;
    g.n8 = round8(nt);
    g.ldv = ld4odd(g.n8);
    g.nb16 = (g.n8 + 15) >> 4;
    g.gpc = (g.nb16 + cs - 1) / cs;
    return g;
}
__host__ __device__ inline size_t lg_panel(const LgGeo &g) {   // N panel or the staged rows of A
    const size_t n = (size_t)16 * g.gpc * g.ldv * 8, a = stage_floats(kLgRows, g.n8) * 4;
    return n > a ? n : a;
}
__host__ __device__ inline size_t lg_smem(int nt, int cs) {
    const LgGeo g = lg_geo(nt, cs);
    return (size_t)kLgN * 8 * 3 + kLgN * 4 + 16 * 4 + (size_t)g.n8 * g.ldv * 8 + (size_t)g.n8 * ld4odd(kLgRows) * 8 +
           lg_panel(g);
}
// Workspace of one matrix: a part of H for every CTA with rows.
__host__ __device__ inline size_t lg_part_bytes(int mt, int nt) {
    const int nb = (round8(nt) + 15) >> 4;
    return (size_t)((mt + kLgRows - 1) / kLgRows) * (nb * (nb + 1) / 2) * 256 * 8;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
// This CTA's shared address as seen in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned remote_smem(const void *ptr, unsigned rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(ptr)), "r"(rank));
    return a;
}
__device__ __forceinline__ void remote_store(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void remote_store(unsigned addr, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Block index -> block row and column (rows of the lower triangle).
__device__ __forceinline__ void lower_block(int b, int &bi, int &bj) {
    bi = 0;
    while (b > bi) { b -= bi + 1; ++bi; }
    bj = b;
}

template <int CS>
__global__ void __launch_bounds__(kRefT, 1) refine_large_kernel(Params p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    const unsigned rank = cluster_rank();
    const int slot = blockIdx.x / CS, slots = gridDim.x / CS;
    double *part = (double *)(p.gws + (size_t)slot * p.gws_stride);
    double *dh = (double *)smem, *de = dh + kLgN, *sig = de + kLgN;
    int *perm = (int *)(sig + kLgN);
    int *flags = perm + kLgN;            // one word of every CTA
    double *V = (double *)(flags + 16);
    for (int64_t idx = slot; idx < p.count; idx += slots) {
        const int mat = p.order ? p.order[idx] : (int)idx;
        if (p.status[mat] != JB_ST_OK) continue;      // the same for the whole cluster
        const jb_matrix_desc d = desc_of(p, mat);
        const bool wide = d.m < d.n;
        const int mt = wide ? d.n : d.m, nt = wide ? d.m : d.n;
        const LgGeo g = lg_geo(nt, CS);
        const int ldv = g.ldv, nt8 = g.n8 >> 3, nblk = g.nb16 * (g.nb16 + 1) / 2;
        constexpr int ldw = 36;                        // ld4odd(kLgRows)
        const int row0 = rank * kLgRows, rows = min(max(mt - row0, 0), kLgRows);
        const int parts = (mt + kLgRows - 1) / kLgRows;
        double *W = V + (size_t)g.n8 * ldv;
        double *Np = W + (size_t)g.n8 * ldw;           // columns 16 gpc rank ..., ld ldv
        float *As = (float *)Np;
        const Stage sg = stage_of(wide, kLgRows, g.n8);
        {
            const float *x = p.x32 + d.x_off;
            for (int c = warp; c < g.n8; c += kRefT / 32)
                for (int i = lane; i < g.n8; i += 32)
                    V[c * ldv + i] = (c < nt && i < nt) ? (double)x[c * nt + i] : 0.0;
        }
        const double tol = p.tol > 0 ? (double)(float)p.tol : (double)(10.0f * Lim<float>::eps());
        const double tol2 = tol * tol;
        const int most = p.max_sweeps < kRefPasses ? p.max_sweeps : kRefPasses;
        int pass = 1;
        bool done = false;
        for (; pass <= most; ++pass) {
            // rows row0 .. of A, zero past the end
            const float *A = (const float *)p.A + d.a_off;
            for (int k = threadIdx.x; k < kLgRows * g.n8; k += kRefT) {
                const int i = wide ? k % kLgRows : k / g.n8, c = wide ? k / kLgRows : k % g.n8;
                const bool in = i < rows && c < nt;
                const float *src = wide ? A + (size_t)c * mt + row0 + i : A + (size_t)(row0 + i) * nt + c;
                cp_async4(As + i * sg.sr + c * sg.sk, in ? src : A, in);
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            ref_mul<4, 1, kRefT / 32, false>(As, sg.sr, sg.sk, V, ldv, W, ldw, g.n8, kLgRows / 8, nt8);
            __syncthreads();
            if (rows > 0) {
                double *mine = part + (size_t)rank * nblk * 256;
                for (int b = warp; b < nblk; b += kRefT / 32) {
                    int bi, bj;
                    lower_block(b, bi, bj);
                    double h0[2][2], h1[2][2];
                    ref_gram(W, ldw, kLgRows, 2 * bi, min(2 * bj, nt8 - 1), nt8, h0);
                    ref_gram(W, ldw, kLgRows, 2 * bi, min(2 * bj + 1, nt8 - 1), nt8, h1);
                    double2 *o = (double2 *)(mine + b * 256 + lane * 8);   // tiles (0,0) (0,1) (1,0) (1,1)
                    o[0] = make_double2(h0[0][0], h0[0][1]);
                    o[1] = make_double2(h1[0][0], h1[0][1]);
                    o[2] = make_double2(h0[1][0], h0[1][1]);
                    o[3] = make_double2(h1[1][0], h1[1][1]);
                }
            }
            cluster_sync();
            // diagonals of H (over the parts) and of E, in every CTA
            for (int c = threadIdx.x; c < nt; c += kRefT) {
                const int b16 = c >> 4, b = b16 * (b16 + 1) / 2 + b16, e = c & 15, f = e & 7;
                const int at = b * 256 + (f * 4 + (f >> 1)) * 8 + (e >> 3) * 6 + (f & 1);
                double sum = 0.0;
                for (int q = 0; q < parts; ++q) sum += part[(size_t)q * nblk * 256 + at];
                dh[c] = sum;
            }
            for (int c = warp; c < nt; c += kRefT / 32) {
                double sum = 0.0;
                for (int i = lane; i < nt; i += 32) sum = fma(V[c * ldv + i], V[c * ldv + i], sum);
                sum = warp_sum(sum);
                if (lane == 0) de[c] = sum - 1.0;
            }
            __syncthreads();
            // this CTA's blocks: the test, and N to the owners of its columns
            int need = 0, wild = 0;
            for (int b = rank + CS * warp; b < nblk; b += CS * (kRefT / 32)) {
                int bi, bj;
                lower_block(b, bi, bj);
                double h[2][2][2] = {}, e0[2][2], e1[2][2];
                for (int q = 0; q < parts; ++q) {
                    const double2 *o = (const double2 *)(part + ((size_t)q * nblk + b) * 256 + lane * 8);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const double2 v = o[t];
                        h[t >> 1][t & 1][0] += v.x;
                        h[t >> 1][t & 1][1] += v.y;
                    }
                }
                ref_gram(V, ldv, g.n8, 2 * bi, min(2 * bj, nt8 - 1), nt8, e0);
                ref_gram(V, ldv, g.n8, 2 * bi, min(2 * bj + 1, nt8 - 1), nt8, e1);
                const unsigned to_c = remote_smem(Np, bj / g.gpc), to_r = remote_smem(Np, bi / g.gpc);
                const int c0 = (bj % g.gpc) * 16, r0 = (bi % g.gpc) * 16;
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int t = 0; t < 2; ++t)
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int rl = a * 8 + lr, cl = t * 8 + 2 * lk + u;
                            const int r = bi * 16 + rl, c = bj * 16 + cl;
                            if (r >= g.n8 || c > r) continue;
                            double nrc = 0.0, ncr = 0.0;
                            if (r < nt) {
                                const double hh = h[a][t][u], ee = c == r ? de[r] : (t ? e1 : e0)[a][u];
                                if (!(fabs(ee) <= kRefOrth)) need = 1;
                                if (c == r) {
                                    nrc = -0.5 * ee;
                                } else {
                                    if (!(hh * hh <= tol2 * dh[r] * dh[c])) need = 1;
                                    const double off = hh - 0.5 * ee * (dh[r] + dh[c]);
                                    const double k = ref_angle(dh[r] * (1.0 - de[r]) - dh[c] * (1.0 - de[c]), off);
                                    if (!(fabs(k) <= 0.25 && fabs(ee) <= 0.1)) wild = 1;
                                    ncr = k - 0.5 * ee;     // N(c, r)
                                    nrc = -k - 0.5 * ee;    // N(r, c)
                                }
                            }
                            remote_store(to_c + ((c0 + cl) * ldv + r) * 8, nrc);
                            if (c < r) remote_store(to_r + ((r0 + rl) * ldv + c) * 8, ncr);
                        }
            }
            const int word = (__syncthreads_or(need) ? 1 : 0) | (__syncthreads_or(wild) ? 2 : 0);
            if (threadIdx.x < CS) remote_store(remote_smem(flags + rank, threadIdx.x), word);
            cluster_sync();
            int all = 0;
#pragma unroll
            for (int q = 0; q < CS; ++q) all |= flags[q];
            if (!(all & 1)) { done = true; break; }
            if ((all & 2) || pass == most) break;
            // second-order term on the diagonal of the owned columns: -sum_i N_ij^2 / 2
            const int own0 = rank * g.gpc * 16, cols = min(max(nt - own0, 0), 16 * g.gpc);
            for (int c = warp; c < cols; c += kRefT / 32) {
                double sum = 0.0;
                for (int i = lane; i < nt; i += 32)
                    if (i != own0 + c) sum = fma(Np[c * ldv + i], Np[c * ldv + i], sum);
                sum = warp_sum(sum);
                if (lane == 0) Np[c * ldv + own0 + c] -= 0.5 * sum;
            }
            __syncthreads();
            // the owned columns of V + V N: 16 x 16 blocks, one a warp and group
            double acc[2][2][2][2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int tc = 2 * (rank * g.gpc + s);     // first column tile
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int t = 0; t < 2; ++t) acc[s][a][t][0] = acc[s][a][t][1] = 0.0;
                if (s < g.gpc && tc < nt8 && 2 * warp < nt8) {
                    const double *x0 = V + lk * ldv + 16 * warp + lr;
                    const double *x1 = V + lk * ldv + (2 * warp + 1 < nt8 ? 16 * warp + 8 : 16 * warp) + lr;
                    const double *y0 = Np + (16 * s + lr) * ldv + lk;
                    const double *y1 = tc + 1 < nt8 ? y0 + 8 * ldv : y0;
#pragma unroll 2
                    for (int k0 = 0; k0 < g.n8; k0 += 4) {
                        const double fa = x0[k0 * ldv], fb = x1[k0 * ldv], f0 = y0[k0], f1 = y1[k0];
                        dmma(acc[s][0][0], fa, f0);
                        dmma(acc[s][1][0], fb, f0);
                        dmma(acc[s][0][1], fa, f1);
                        dmma(acc[s][1][1], fb, f1);
                    }
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (2 * warp + a < nt8 && tc + t < nt8) {
                                const double *v = V + ((tc + t) * 8 + 2 * lk) * ldv + (2 * warp + a) * 8 + lr;
                                acc[s][a][t][0] += v[0];
                                acc[s][a][t][1] += v[ldv];
                            }
                }
            }
            cluster_sync();    // every CTA is done with the old V
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int tc = 2 * (rank * g.gpc + s);
                if (s < g.gpc && tc < nt8 && 2 * warp < nt8) {
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (2 * warp + a < nt8 && tc + t < nt8) {
                                const double *v = V + ((tc + t) * 8 + 2 * lk) * ldv + (2 * warp + a) * 8 + lr;
#pragma unroll
                                for (int q = 0; q < CS; ++q) {
                                    const unsigned to = remote_smem(v, q);
                                    remote_store(to, acc[s][a][t][0]);
                                    remote_store(to + ldv * 8, acc[s][a][t][1]);
                                }
                            }
                }
            }
            cluster_sync();
        }
        // sigma, the stable descending order and the cut (primitives.py:356-366), in every CTA
        int st = JB_ST_OK;
        if (done) {
            for (int j = threadIdx.x; j < nt; j += kRefT) sig[j] = sqrt(dh[j]);
            __syncthreads();
            int below = 0;
            for (int j = threadIdx.x; j < nt; j += kRefT) {
                const double sj = sig[j];
                int rnk = 0;
                double smax = 0.0;
                for (int i = 0; i < nt; ++i) {
                    const double si = sig[i];
                    rnk += (si > sj) || (si == sj && i < j);
                    smax = fmax(smax, si);
                }
                const int npref = nt + (nt & 1);
                if (!(sj > Lim<double>::eps() * (mt > npref ? mt : npref) * smax)) below = 1;
                perm[rnk] = j;
                dh[j] = 1.0 / sj;
            }
            if (__syncthreads_or(below)) done = false;   // columns to complete: not here
        }
        int bad = 0;
        if (!done) {
            st = kPending;
        } else {
            if (rank == 0 && threadIdx.x < d.rank) {
                const float o = (float)sig[perm[threadIdx.x]];
                if (!isfinite(o)) bad = 1;
                ((float *)p.S + d.s_off)[threadIdx.x] = o;
            }
            if (!(d.flags & JB_VALUES_ONLY)) {
                float *U = (float *)p.U + d.u_off, *Vh = (float *)p.Vh + d.v_off;
                // W's rows of this CTA: rows of U, or columns of Vh of a wide matrix
                for (int k = threadIdx.x; k < rows * d.rank; k += kRefT) {
                    const int i = wide ? k % rows : k / d.rank, r = wide ? k / rows : k % d.rank, c = perm[r];
                    const float o = (float)(W[c * ldw + i] * dh[c]);
                    if (!isfinite(o)) bad = 1;
                    if (wide) Vh[(size_t)r * mt + row0 + i] = o;
                    else U[(size_t)(row0 + i) * d.rank + r] = o;
                }
                // V's part: nt x rank entries shared out over the cluster
                for (int k = rank * kRefT + threadIdx.x; k < nt * d.rank; k += CS * kRefT) {
                    const int i = wide ? k / d.rank : k % nt, r = wide ? k % d.rank : k / nt;
                    const float o = (float)V[perm[r] * ldv + i];
                    if (!isfinite(o)) bad = 1;
                    if (wide) U[(size_t)i * d.rank + r] = o;
                    else Vh[(size_t)r * nt + i] = o;
                }
            }
        }
        const int word = __syncthreads_or(bad);
        if (threadIdx.x == 0) remote_store(remote_smem(flags + 8 + rank, 0), word);
        cluster_sync();   // also: no CTA starts on the next matrix while another reads this one's
        if (rank == 0 && threadIdx.x == 0) {
            for (int q = 0; q < CS; ++q)
                if (flags[8 + q]) st = JB_ST_NONFINITE_OUT;
            p.status[mat] = st;
            if (st == kPending) atomicAdd(p.n_pending, 1);
            else p.sweeps[mat] += pass;
        }
    }
}

}  // namespace jb
