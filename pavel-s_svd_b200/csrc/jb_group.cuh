// jb_group.cuh - one-sided Jacobi sweeps with GL lanes a block pair, W and V in
// registers, in the input's own arithmetic (FP32, FP64, complex of either).
//
// The columns of [W; V] are split into nb blocks of B; group g of GL lanes
// holds the blocks at positions (g, nb - 1 - g) of a circle-method tournament
// over blocks, lane gl the elements of the 16-byte chunks gl, gl + GL, ... of
// all 2B columns.  A sweep pairs the columns inside each block, then has nb - 1
// block rounds of B steps that pair x_i with y_(i+j); every column pair once,
// as the reference's round-robin sweep (svdbench/standalone/primitives.py:
// 328-351).  All groups of a warp share the instructions of a step's fixed
// part -- reductions, rotation parameters, broadcasts -- which bounds a step
// when a whole warp works on one block pair (jb_regblock.cuh: 39 instructions a
// column pair at 64 x 32; here 16).
//
// Columns are kept scaled, w = d * (the register column): a rotation is then
// x - a y, y + b x with both scales multiplied by c, half the arithmetic of
// the plain form (Gentleman's rotation).  Scales start at 1 every sweep and
// shrink by at most sqrt(2) a rotation; they are FP64 also for FP32 input,
// with c = 1 - t^2 / (1 + t^2 + sqrt(1 + t^2)): a c rounded to FP32 loses t^2 <
// 6e-8 of every small rotation, always to the same side.  The three dot products of a pair are
// exact sums each time, the active test and the angle are the reference's
// (primitives.py:334-347); the null-column floor eps^2 max ||w_j||^2 takes the
// norms at the start of the sweep (the reference's: of the round).
//
// EIG: the two-sided Jacobi of a Hermitian H (primitives.py:370-427) in the same
// form: W = H V and V are rotated together, and the entries of G = V^H H V that a
// rotation needs are the dot products v_p^H w_p, v_q^H w_q, v_p^H w_q -- no row
// rotations, and G itself is never formed.  A pair is active when |g_pq| > tol
// max|G| (the reference's absolute criterion; max|G| is that of H in the first
// sweep, then the largest |g_pp| at the start of the sweep).
#pragma once
#include "jb_device.cuh"
#include "jb_regblock.cuh"

namespace jb {

// R: float or double; NC: 1 real, 2 complex; rows of W and V a lane.
template <typename R, int NC, int GL, int B, int RW, int RV>
struct GroupCfg {
    static constexpr int CH = 16 / sizeof(R);            // elements of a chunk
    static constexpr int EW = RW * NC, ET = (RW + RV) * NC;   // elements of a lane: W, both
    static_assert(EW % CH == 0 && ET % CH == 0, "whole chunks");
    static constexpr int MC = GL * RW, NCOLS = GL * RV;  // rows of W and V that fit
    static constexpr int VOFF = GL * EW;                 // V's elements of a column after W's
    static constexpr int LD = GL * ET + CH;              // a column in shared memory (16 bytes of padding)
};

template <int GL, typename R, int NV>
__device__ __forceinline__ void lanes_reduce_scatter(R (&x)[NV], int lane) {
    constexpr int L = Log2<NV>::value;
#pragma unroll
    for (int s = 0; s < L; ++s) {
        const int h = NV >> (s + 1);
        const int o = (GL / 2) >> s;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const R send = up ? x[k] : x[k + h];
            const R keep = up ? x[k + h] : x[k];
            x[k] = keep + __shfl_xor_sync(FULL, send, o);
        }
    }
#pragma unroll
    for (int o = (GL / 2) >> L; o >= 1; o >>= 1) x[0] += __shfl_xor_sync(FULL, x[0], o);
}

// Tangent of the reference's rotation for |apq| = a >= 0; false (t = 0) for an
// inactive pair.
// FP32: from approximate reciprocals (an error of a few ulp in t only leaves
// |apq| a few ulp of itself).
// FP64: accurate to rounding, so that one rotation leaves the pair
// orthogonal to rounding level as the reference's FP64 arithmetic does (an
// FP32 angle leaves a ratio ~1e-7 of the one it removed, near 10 eps in the
// last rotating sweep, and costs a sweep).  With the exponent-scaled dd = |d|
// scl, aa = 2a scl (max of the two in [1, 2)), t is the positive root of g(t) =
// aa t^2 + 2 dd t - aa: the FP32 estimate, then two Newton steps t -= g(t) /
// g'(t) with g'/2 = aa t + dd >= 1/2 inverted once in FP32 (each step
// multiplies the error by ~1e-7; g(t) is evaluated to rounding of its largest
// term, ~aa, so small angles keep their relative accuracy).
__device__ __forceinline__ bool jacobi_tan(float app, float aqq, float a, float tol2, float floor_, float &t) {
    const float a2 = a * a, prod = app * aqq;
    t = 0.f;
    if (!(a2 > tol2 * prod && fminf(app, aqq) > floor_)) return false;
    const float d = aqq - app;
    const float h = fmaf(d, d, 4.f * a2);
    t = copysignf(__fdividef(2.f * a, fabsf(d) + h * rsqrtf(h)), d);
    return true;
}
__device__ __forceinline__ bool eigen_tan(double app, double aqq, double a, double threshold, double &t) {
    t = 0.0;
    if (!(a > threshold)) return false;
    const double d = aqq - app, a2 = 2.0 * a;
    const int ex = (__double2hiint(fmax(fabs(d), a2)) >> 20) & 0x7ff;
    const double scl = __hiloint2double((2046 - ex) << 20, 0);
    const double dd = fabs(d) * scl, aa = a2 * scl;
    const float df = (float)dd, af = (float)aa;
    const float hf = fmaf(df, df, af * af);
    t = (double)__fdividef(af, df + hf * rsqrtf(hf));
    const double r = 0.5 * (double)__frcp_rn((float)fma(aa, t, dd));
#pragma unroll
    for (int k = 0; k < 2; ++k) t -= fma(aa * t, t, fma(2.0 * dd, t, -aa)) * r;
    if (d < 0.0) t = -t;
    return true;
}
__device__ __forceinline__ bool jacobi_tan(double app, double aqq, double a, double tol2, double floor_, double &t) {
    const bool active = a * a > tol2 * (app * aqq) && fmin(app, aqq) > floor_;
    return eigen_tan(app, aqq, active ? a : 0.0, 0.0, t);
}
// c = 1 / sqrt(1 + t2): FP32 from 1 - c with its own relative precision, FP64
// the FP32 estimate and two Newton steps.
__device__ __forceinline__ double cosine(float t2) {
    const float x = 1.f + t2;
    return 1.0 - (double)__fdividef(t2, fmaf(x, rsqrtf(x), x));
}
__device__ __forceinline__ double cosine(double t2) {
    const double x = 1.0 + t2, hx = -0.5 * x;
    double c = (double)rsqrtf((float)x);
#pragma unroll
    for (int k = 0; k < 2; ++k) c *= fma(hx, c * c, 1.5);
    return c;
}
// 1 / x for a scale in (2^-64, 1], to rounding.
__device__ __forceinline__ float inv_scale(float x) {
    const float r = __fdividef(1.f, x);
    return r * fmaf(-x, r, 2.f);
}
__device__ __forceinline__ double inv_scale(double x) {
    double r = (double)__fdividef(1.f, (float)x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}
// 1 / sqrt(x), x normal: to rounding (FP64) or an ulp or two (FP32).
__device__ __forceinline__ float rsqrt_of(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrt_of(double x) {
    // FP32 estimate of the mantissa in [1, 4), two Newton steps
    const int ex = ((__double2hiint(x) >> 20) & 0x7fe) - 1022;   // even
    const double scl = __hiloint2double((1023 - ex) << 20, 0), xs = x * scl;
    double r = (double)rsqrtf((float)xs);
#pragma unroll
    for (int k = 0; k < 2; ++k) r *= fma(-0.5 * xs, r * r, 1.5);
    return r * __hiloint2double((1023 - (ex >> 1)) << 20, 0);
}

template <typename R, int NC, int GL, int B, int RW, int RV, bool EIG = false>
struct GroupTile {
    using C = GroupCfg<R, NC, GL, B, RW, RV>;
    static_assert(B <= 2, "blocks of one or two columns");
    R w[2 * B][C::ET];
    double dx, dy;   // scales of the lane's pair (x_i, y_i), i = (lane in group) / (GL / B)

    // x <- x - conj(a) y, y <- y + b x (b along a); real: ai, bi unused
    __device__ __forceinline__ void rotate(int p, int q, R ar, R ai, R br, R bi) {
        if constexpr (NC == 1 && sizeof(R) == 4) {
            const float2 na = make_float2(-ar, -ar), pb = make_float2(br, br);
#pragma unroll
            for (int e = 0; e < C::ET; e += 2) {
                const float2 u = make_float2(w[p][e], w[p][e + 1]), v = make_float2(w[q][e], w[q][e + 1]);
                const float2 u2 = __ffma2_rn(na, v, u), v2 = __ffma2_rn(pb, u, v);
                w[p][e] = u2.x; w[p][e + 1] = u2.y;
                w[q][e] = v2.x; w[q][e + 1] = v2.y;
            }
        } else if constexpr (NC == 1) {
#pragma unroll
            for (int e = 0; e < C::ET; ++e) {
                const R x = w[p][e], y = w[q][e];
                w[p][e] = dfma(-ar, y, x);
                w[q][e] = dfma(br, x, y);
            }
        } else if constexpr (sizeof(R) == 4) {
            const float2 a1 = make_float2(-ar, -ar), a2 = make_float2(-ai, ai);
            const float2 b1 = make_float2(br, br), b2 = make_float2(-bi, bi);
#pragma unroll
            for (int e = 0; e < C::ET; e += 2) {
                const float2 u = make_float2(w[p][e], w[p][e + 1]), v = make_float2(w[q][e], w[q][e + 1]);
                const float2 us = make_float2(u.y, u.x), vs = make_float2(v.y, v.x);
                const float2 u2 = __ffma2_rn(a1, v, __ffma2_rn(a2, vs, u));
                const float2 v2 = __ffma2_rn(b1, u, __ffma2_rn(b2, us, v));
                w[p][e] = u2.x; w[p][e + 1] = u2.y;
                w[q][e] = v2.x; w[q][e + 1] = v2.y;
            }
        } else {
#pragma unroll
            for (int e = 0; e < C::ET; e += 2) {
                const R xr = w[p][e], xi = w[p][e + 1], yr = w[q][e], yi = w[q][e + 1];
                w[p][e] = dfma(-ar, yr, dfma(-ai, yi, xr));
                w[p][e + 1] = dfma(-ar, yi, dfma(ai, yr, xi));
                w[q][e] = dfma(br, xr, dfma(-bi, xi, yr));
                w[q][e + 1] = dfma(br, xi, dfma(bi, xr, yi));
            }
        }
    }
    __device__ __forceinline__ void scale(int p, R s) {
#pragma unroll
        for (int e = 0; e < C::ET; ++e) w[p][e] *= s;
    }
    // ||w_p||^2, or v_p^H w_p
    __device__ __forceinline__ R norm2(int p) const {
        constexpr int O = EIG ? C::EW : 0;
        R a = 0, b = 0;
#pragma unroll
        for (int e = 0; e < C::EW; e += 2) {
            if constexpr (sizeof(R) == 4) {
                fma2(a, b, w[p][O + e], w[p][O + e + 1], w[p][e], w[p][e + 1]);
            } else {
                a = dfma(w[p][O + e], w[p][e], a);
                b = dfma(w[p][O + e + 1], w[p][e + 1], b);
            }
        }
        return a + b;
    }
    // re and im of w_p^H w_q, or v_p^H w_q
    __device__ __forceinline__ void dot(int p, int q, R &re, R &im) const {
        constexpr int O = EIG ? C::EW : 0;
        R a = 0, b = 0, c = 0, d = 0;
#pragma unroll
        for (int e = 0; e < C::EW; e += 2) {
            if constexpr (sizeof(R) == 4) {
                fma2(a, b, w[p][O + e], w[p][O + e + 1], w[q][e], w[q][e + 1]);
            } else {
                a = dfma(w[p][O + e], w[q][e], a);
                b = dfma(w[p][O + e + 1], w[q][e + 1], b);
            }
            if constexpr (NC == 2) {
                if constexpr (sizeof(R) == 4) {
                    fma2(c, d, w[p][O + e], w[p][O + e + 1], w[q][e + 1], w[q][e]);
                } else {
                    c = dfma(w[p][O + e], w[q][e + 1], c);
                    d = dfma(w[p][O + e + 1], w[q][e], d);
                }
            }
        }
        re = a + b;
        im = c - d;
    }

    // One step: B disjoint pairs of each group.  INTRA pairs the two columns of
    // each block (scales 1 before), otherwise x_i with y_i.  EIG: floor_ is the
    // threshold of |g_pq|.
    template <bool INTRA>
    __device__ __forceinline__ void step(R tol2, R floor_, int &fl, int lane) {
        constexpr int LB = Log2<B>::value, LG = Log2<GL>::value;
        R pa[B], pb[B], pr[B], pi[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int p = pair_p<INTRA, B>(i), q = pair_q<INTRA, B>(i);
            pa[i] = norm2(p);
            pb[i] = norm2(q);
            dot(p, q, pr[i], pi[i]);
        }
        lanes_reduce_scatter<GL>(pa, lane);
        lanes_reduce_scatter<GL>(pb, lane);
        lanes_reduce_scatter<GL>(pr, lane);
        if constexpr (NC == 2) lanes_reduce_scatter<GL>(pi, lane);
        // complex FP32: the squares of apq scaled by 2^80, away from denormals
        constexpr R S = NC == 2 && sizeof(R) == 4 ? R(1048576) : R(1);
        R app = pa[0], aqq = pb[0], re = pr[0], im = NC == 2 ? pi[0] : R(0);
        R sx = S, sy = S;
        if constexpr (!INTRA) { sx *= (R)dx; sy *= (R)dy; }
        app *= sx * sx;
        aqq *= sy * sy;
        re *= sx * sy;
        if (NC == 2) im *= sx * sy;
        R t, tr, ti = 0;
        bool active;
        if constexpr (NC == 2) {
            // t e^(i phi), phi the phase of apq
            const R g2 = dfma(re, re, im * im), ig = rsqrt_of(fmax(g2, Lim<R>::tiny()));
            if constexpr (EIG) active = eigen_tan(app, aqq, g2 * ig, floor_, t);
            else active = jacobi_tan(app, aqq, g2 * ig, tol2, floor_ * S * S, t);
            tr = active ? t * ig * re : R(0);
            ti = active ? t * ig * im : R(0);
        } else {
            if constexpr (EIG) active = eigen_tan(app, aqq, dabs(re), floor_, t);
            else active = jacobi_tan(app, aqq, dabs(re), tol2, floor_, t);
            tr = re < R(0) ? -t : t;
        }
        if (active) fl = 1;
        if (!__any_sync(FULL, active)) return;
        const double c = cosine(NC == 2 ? dfma(tr, tr, ti * ti) : tr * tr);
        R ar = tr, ai = ti, br = tr, bi = ti;
        if constexpr (!INTRA) {
            const R f = sy * inv_scale(sx), g = sx * inv_scale(sy);
            ar *= f; ai *= f;
            br *= g; bi *= g;
            dx *= c;
            dy *= c;
        } else {   // columns 0, 1 of x are pair 0, those of y pair 1
            dx = __shfl_sync(FULL, c, lane & ~(GL - 1));
            dy = __shfl_sync(FULL, c, (lane & ~(GL - 1)) | (GL / 2));
        }
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int src = (lane & ~(GL - 1)) | (i << (LG - LB));
            const R xr = __shfl_sync(FULL, ar, src), yr = __shfl_sync(FULL, br, src);
            R xi = 0, yi = 0;
            if constexpr (NC == 2) { xi = __shfl_sync(FULL, ai, src); yi = __shfl_sync(FULL, bi, src); }
            rotate(pair_p<INTRA, B>(i), pair_q<INTRA, B>(i), xr, xi, yr, yi);
        }
    }
    __device__ __forceinline__ void shift_y(int lane) {
        if constexpr (B > 1) {
            dy = __shfl_sync(FULL, dy, (lane & ~(GL - 1)) | ((lane + GL / B) & (GL - 1)));
#pragma unroll
            for (int e = 0; e < C::ET; ++e) {
                const R f = w[B][e];
#pragma unroll
                for (int i = 0; i < B - 1; ++i) w[B + i][e] = w[B + i + 1][e];
                w[2 * B - 1][e] = f;
            }
        }
    }
    template <bool STORE>
    __device__ __forceinline__ void exchange(R *area, int X, int Y, int gl) {
#pragma unroll
        for (int c = 0; c < 2 * B; ++c) {
            R *col = area + (c < B ? X * B + c : Y * B + (c - B)) * C::LD + gl * C::CH;
#pragma unroll
            for (int k = 0; k < C::ET / C::CH; ++k) {
                if constexpr (sizeof(R) == 4) {
                    float4 *p = (float4 *)(col + k * GL * 4);
                    if (STORE) *p = make_float4(w[c][4 * k], w[c][4 * k + 1], w[c][4 * k + 2], w[c][4 * k + 3]);
                    else {
                        const float4 v = *p;
                        w[c][4 * k] = v.x; w[c][4 * k + 1] = v.y; w[c][4 * k + 2] = v.z; w[c][4 * k + 3] = v.w;
                    }
                } else {
                    double2 *p = (double2 *)(col + k * GL * 2);
                    if (STORE) *p = make_double2(w[c][2 * k], w[c][2 * k + 1]);
                    else {
                        const double2 v = *p;
                        w[c][2 * k] = v.x; w[c][2 * k + 1] = v.y;
                    }
                }
            }
        }
    }
};

template <int THREADS>
__device__ __forceinline__ void team_sync() {
    if constexpr (THREADS == 32) __syncwarp();
    else __syncthreads();
}

// Sweeps over the n columns in `area` (column c at c * LD: W then V; columns up
// to the block grid zero) until one finds no active pair; the rotated columns
// are left there, at scale 1.  scales: npb doubles of shared memory; red: 32
// doubles.  All threads of the CTA call it.  Returns the sweeps taken.
// EIG: max|H| is given as scale0.
template <typename R, int NC, int GL, int B, int RW, int RV, int THREADS, bool EIG = false>
__device__ int group_sweeps(R *area, int n, R tol, int max_sweeps, double *scales, double *red, bool &converged,
                            R scale0 = R(0)) {
    constexpr int LB = Log2<B>::value, LG = Log2<GL>::value;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & (GL - 1);
    const int group = threadIdx.x / GL, li = gl >> (LG - LB), base = lane & ~(GL - 1);
    const int nb = 2 * ((n + 2 * B - 1) / (2 * B));
    const bool act = group < nb / 2, wact = warp * (32 / GL) < nb / 2;
    GroupTile<R, NC, GL, B, RW, RV, EIG> t;
    int X = act ? group : 0, Y = act ? nb - 1 - group : 0;
    if (act) {
        t.template exchange<false>(area, X, Y, gl);
    } else {
#pragma unroll
        for (int c = 0; c < 2 * B; ++c)
#pragma unroll
            for (int e = 0; e < GroupCfg<R, NC, GL, B, RW, RV>::ET; ++e) t.w[c][e] = R(0);
    }
    const R tol2 = tol * tol;
    converged = false;
    int sweep = 1;
    t.dx = t.dy = 1.0;
#pragma unroll 1
    for (; sweep <= max_sweeps; ++sweep) {
        R mx = R(0);
        if (wact) {
#pragma unroll
            for (int c = 0; c < 2 * B; ++c) {
                R s[1] = {t.norm2(c)};
                lanes_reduce_scatter<GL>(s, lane);
                mx = fmax(mx, EIG ? dabs(s[0]) : s[0]);
            }
        }
        mx = warp_max(mx);
        if constexpr (THREADS > 32) {
            if (lane == 0) red[warp] = (double)mx;
            __syncthreads();
            double gm = 0.0;
#pragma unroll
            for (int w = 0; w < THREADS / 32; ++w) gm = fmax(gm, red[w]);
            mx = (R)gm;
        }
        const R floor_ = EIG ? tol * (sweep == 1 ? scale0 : mx) : Lim<R>::eps() * Lim<R>::eps() * mx;
        int fl = 0;
        if (wact) {
            if constexpr (B == 2) t.template step<true>(tol2, floor_, fl, lane);
        }
#pragma unroll 1
        for (int br = 0; br < nb - 1; ++br) {
            if (br > 0 || sweep > 1) {
                if (act) {
                    t.template exchange<true>(area, X, Y, gl);
                    if ((gl & (GL / B - 1)) == 0) {
                        scales[X * B + li] = t.dx;
                        scales[Y * B + li] = t.dy;
                    }
                }
                team_sync<THREADS>();
                if (act) {
                    if (X > 0) X = X == 1 ? nb - 1 : X - 1;
                    Y = Y == 1 ? nb - 1 : Y - 1;
                    t.template exchange<false>(area, X, Y, gl);
                    t.dx = scales[X * B + li];
                    t.dy = scales[Y * B + li];
                }
            }
            if (wact) {
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    t.template step<false>(tol2, floor_, fl, lane);
                    t.shift_y(lane);
                }
            }
        }
        if (wact) {   // back to scale 1
#pragma unroll
            for (int i = 0; i < B; ++i) {
                const R sx = __shfl_sync(FULL, (R)t.dx, base | (i << (LG - LB)));
                const R sy = __shfl_sync(FULL, (R)t.dy, base | (i << (LG - LB)));
                t.scale(i, sx);
                t.scale(B + i, sy);
            }
            t.dx = t.dy = 1.0;
        }
        const bool any = THREADS == 32 ? __any_sync(FULL, fl) : __syncthreads_or(fl);
        if (!any) { converged = true; break; }
    }
    team_sync<THREADS>();
    if (act) t.template exchange<true>(area, X, Y, gl);
    team_sync<THREADS>();
    return converged ? sweep : max_sweeps;
}

}  // namespace jb
