// jb_null.cu - null-space completion of U on the GPU
// (svdbench/standalone/primitives.py:430-455, complete_null_columns; used by
// complete_basis :458-467 and by _finish_columns, solvers.py:18-21).
//
// For every matrix of a batch U (batch x m x n, row-major) and its keep mask
// (batch x n bytes): the columns not kept are replaced, in ascending column
// order, by unit vectors orthogonal to all columns before them.  Per missing
// column, as the reference: idx = the first row of largest leftover leverage
// 1 - sum_c |u_ic|^2 (over the kept and the already completed columns),
// v = e_idx projected out against those columns, v / ||v||; ||v|| < 10 eps
// of the dtype fails the matrix (JB_ST_NULL_FAILED, primitives.py:451-452).
//
// B200 form.  The columns that count (kept, then completed ones in the order
// they are made) are packed into a work matrix X (m x a, row stride n), so
// every product reads a contiguous row prefix.  U^H e_idx is row idx of X,
// so the first projection is row-local: v_i = delta_{i,idx} - X_i . conj(X_idx).
// The leverage is kept per row in FP64 and lowered by |v_i|^2 after each new
// column; products accumulate in FP64 (complex: FP64 pairs).
//   * Many matrices (team of one CTA per matrix): the second projection
//     always runs, as in the reference.
//   * Few large matrices: one team of CTAs (about 64 rows each, at most one
//     per SM, cooperative launch) handles one matrix after another.  The
//     first projection's length^2 equals the pivot's leverage (v = P e_idx,
//     P the projector onto the complement), so while that leverage is at
//     least 1/2 a column costs one grid-wide barrier: v is normalised by it
//     directly (Kahan-Parlett "twice is enough": v is then orthogonal to the
//     columns to working accuracy and needs no second projection).  Below
//     1/2 the second projection runs, with the norm reduced over the team.
// Every barrier wait is bounded (about two seconds of globaltimer); a wait
// that runs out marks the team's matrix JB_ST_TIMEOUT and the CTAs return.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include "jacobi_b200.h"

namespace jb {
namespace nul {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr unsigned long long kWaitNs = 2000000000ull;

struct cf { float x, y; };
struct cd { double x, y; };

// Element traits: storage type S, FP64 accumulation type A.
template <typename S> struct Tr;
template <> struct Tr<float> {
    using A = double;
    static constexpr bool cplx = false;
    static constexpr double eps = 1.1920928955078125e-07;
    __device__ static A zero() { return 0.0; }
    __device__ static A ld(const float *p) { return (double)*p; }
    __device__ static A ldcg(const float *p) { return (double)__ldcg(p); }
    __device__ static void st(float *p, A v) { *p = (float)v; }
    __device__ static A fma_(A acc, A x, A y) { return fma(x, y, acc); }
    __device__ static double norm2(A x) { return x * x; }
    __device__ static A scale(A x, double s) { return x * s; }
    __device__ static A sub(A x, A y) { return x - y; }
    __device__ static A add(A x, A y) { return x + y; }
    __device__ static A conj(A x) { return x; }
    __device__ static A ldcgA(const A *p) { return __ldcg(p); }
    __device__ static A unit() { return 1.0; }
    __device__ static A shfl_sum(A v) {
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
};
template <> struct Tr<double> {
    using A = double;
    static constexpr bool cplx = false;
    static constexpr double eps = 2.220446049250313e-16;
    __device__ static A zero() { return 0.0; }
    __device__ static A ld(const double *p) { return *p; }
    __device__ static A ldcg(const double *p) { return __ldcg(p); }
    __device__ static void st(double *p, A v) { *p = v; }
    __device__ static A fma_(A acc, A x, A y) { return fma(x, y, acc); }
    __device__ static double norm2(A x) { return x * x; }
    __device__ static A scale(A x, double s) { return x * s; }
    __device__ static A sub(A x, A y) { return x - y; }
    __device__ static A add(A x, A y) { return x + y; }
    __device__ static A conj(A x) { return x; }
    __device__ static A ldcgA(const A *p) { return __ldcg(p); }
    __device__ static A unit() { return 1.0; }
    __device__ static A shfl_sum(A v) {
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
};
template <typename S, typename R> struct TrC {
    using A = cd;
    static constexpr bool cplx = true;
    __device__ static A zero() { return {0.0, 0.0}; }
    __device__ static A ld(const S *p) { return {(double)p->x, (double)p->y}; }
    __device__ static A ldcg(const S *p) {
        const R *q = (const R *)p;
        return {(double)__ldcg(q), (double)__ldcg(q + 1)};
    }
    __device__ static void st(S *p, A v) { p->x = (R)v.x; p->y = (R)v.y; }
    __device__ static A fma_(A acc, A x, A y) {                          // acc + x * y
        return {fma(x.x, y.x, fma(-x.y, y.y, acc.x)), fma(x.x, y.y, fma(x.y, y.x, acc.y))};
    }
    __device__ static double norm2(A x) { return x.x * x.x + x.y * x.y; }
    __device__ static A scale(A x, double s) { return {x.x * s, x.y * s}; }
    __device__ static A sub(A x, A y) { return {x.x - y.x, x.y - y.y}; }
    __device__ static A add(A x, A y) { return {x.x + y.x, x.y + y.y}; }
    __device__ static A conj(A x) { return {x.x, -x.y}; }
    __device__ static A ldcgA(const A *p) { return {__ldcg(&p->x), __ldcg(&p->y)}; }
    __device__ static A unit() { return {1.0, 0.0}; }
    __device__ static A shfl_sum(A v) {
        for (int o = 16; o; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        return v;
    }
};
template <> struct Tr<cf> : TrC<cf, float> { static constexpr double eps = 1.1920928955078125e-07; };
template <> struct Tr<cd> : TrC<cd, double> { static constexpr double eps = 2.220446049250313e-16; };

struct Slot {            // one CTA's contribution to a team-wide reduction
    double val;          // norm^2 partial, or the CTA's best leverage
    int64_t idx;         // row of the best leverage (first on ties)
};

struct Params {
    void *U;
    const uint8_t *keep;
    int32_t *status;
    int64_t batch, m, n;
    unsigned char *ws;   // per-team areas of team_bytes each
    size_t team_bytes;
    int G;               // CTAs per team (1: every CTA is a team)
    int always_reorth;
    int blocked;         // team path, real types: the blocked pass may run (block_pass)
};

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Team-wide barrier.  G == 1: the CTA barrier.  G > 1: one counter of
// arrivals over the whole (co-resident, cooperative) grid, waited on until the
// generation's last arrival; a few ns a CTA on one L2 word, where two levels of
// counters cost three dependent atomics (3.3 us a barrier over 128 CTAs; 1.9
// with the one counter).  Waits are bounded; returns false once any CTA of the
// team gave up.  bar[0] arrivals, bar[2] error flag (the area is zeroed before
// the launch).
__device__ __forceinline__ bool team_sync(unsigned *bar, int G) {
    __syncthreads();
    if (G == 1) return true;
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        volatile unsigned *vbar = bar;
        volatile int *verr = (volatile int *)(bar + 2);
        __threadfence();
        const unsigned target = (atomicAdd(bar, 1u) / (unsigned)G + 1u) * (unsigned)G;
        int ok = 1;
        const unsigned long long t0 = gtimer();
        while ((int)(*vbar - target) < 0) {
            if (gtimer() - t0 > kWaitNs) {
                ok = 0;
                atomicExch((int *)(bar + 2), 1);
                break;
            }
        }
        __threadfence();
        s_ok = ok && !*verr;
    }
    __syncthreads();
    return s_ok != 0;
}

// Best (largest val, then smallest idx) of the CTA's candidates; result in
// thread 0.  `red` holds kWarps slots.
__device__ __forceinline__ Slot cta_argmax(double best, int64_t bidx, Slot *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int64_t oi = __shfl_xor_sync(0xffffffffu, bidx, o);
        if (ob > best || (ob == best && oi < bidx)) { best = ob; bidx = oi; }
    }
    if (lane == 0) red[warp] = {best, bidx};
    __syncthreads();
    Slot s = red[0];
    if (threadIdx.x == 0)
        for (int w = 1; w < kWarps; ++w)
            if (red[w].val > s.val || (red[w].val == s.val && red[w].idx < s.idx)) s = red[w];
    __syncthreads();
    return s;
}

__device__ __forceinline__ double cta_sum(double v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kWarps; ++w) s += red[w];
    __syncthreads();
    return s;
}

// Team-wide reductions over the G slots, read by warp 0 only (one L2 read
// per slot per CTA) and broadcast through shared memory.
__device__ __forceinline__ Slot team_argmax(const Slot *slots, int G, bool team, Slot *s_slot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        double best = -1e300;
        int64_t bidx = 0;
        for (int q = lane; q < G; q += 32) {
            const double v = team ? __ldcg(&slots[q].val) : slots[q].val;
            const int64_t i = team ? __ldcg(&slots[q].idx) : slots[q].idx;
            if (v > best || (v == best && i < bidx)) { best = v; bidx = i; }
        }
        for (int o = 16; o; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int64_t oi = __shfl_xor_sync(0xffffffffu, bidx, o);
            if (ob > best || (ob == best && oi < bidx)) { best = ob; bidx = oi; }
        }
        if (lane == 0) *s_slot = {best, bidx};
    }
    __syncthreads();
    const Slot r = *s_slot;
    __syncthreads();
    return r;
}

// Sum of slots[q].val over q < G in a fixed order (the same value in every
// CTA): lane-strided partial sums combined by a fixed butterfly.
__device__ __forceinline__ double team_sum(const Slot *slots, int G, bool team, double *s_val) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        double v = 0.0;
        for (int q = lane; q < G; q += 32) v += team ? __ldcg(&slots[q].val) : slots[q].val;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) *s_val = v;
    }
    __syncthreads();
    const double r = *s_val;
    __syncthreads();
    return r;
}

// Row stride of the packed columns X: a multiple of 16 bytes, so that every
// row starts aligned for 16-byte vector loads.
__host__ __device__ inline int64_t x_stride(int64_t n, int esz) {
    const int64_t v = 16 / esz;
    return (n + v - 1) / v * v;
}

// Blocked pass of the team path (block_pass): the most rows the CTAs publish
// for a block, the most of them it takes as candidates (their projector block
// then fits in shared memory), columns per block at most, and the most rows a
// CTA may hold for it (its local sort).
constexpr int kPubMax = 256;
constexpr int kCand = 128;
constexpr int kBlk = 32;
constexpr int kSortMax = 1024;
static_assert(kCand == kThreads / 4 && kCand % 32 == 0 && kPubMax == kThreads / 2 && kBlk == 32 && kSortMax >= 64, "blocked pass sizes");

// Per-team workspace layout (byte offsets from the team's base).  X, the
// packed columns, and the blocked pass's areas exist only for multi-CTA teams:
// cand (every CTA's best rows), bm (the candidate block of the projector,
// kCand^2), bl (kBlk^2 triangular factor), bp (pivot rows), bv (pivot
// leverages), bmeta.
struct Layout {
    size_t x, lev, y, part, cmap, slots, bar, cand, bm, bl, bp, bv, bmeta, total;
};
__host__ __device__ inline size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }
__host__ __device__ inline Layout layout(int64_t m, int64_t n, int esz, int asz, int G) {
    Layout L;
    size_t o = 0;
    const bool team = G > 1;
    L.x = o;     o += team ? al256((size_t)m * x_stride(n, esz) * esz) : 0;
    L.lev = o;   o += al256((size_t)m * 8);
    L.y = o;     o += al256((size_t)n * asz);
    L.part = o;  o += team ? al256((size_t)G * n * asz) : 0;
    L.cmap = o;  o += al256((size_t)n * 4);
    L.slots = o; o += al256((size_t)2 * G * sizeof(Slot));
    L.bar = o;   o += 256;
    L.cand = o;  o += team ? al256((size_t)kPubMax * sizeof(Slot)) : 0;
    L.bm = o;    o += team ? al256((size_t)kCand * kCand * 8) : 0;
    L.bl = o;    o += team ? al256((size_t)kBlk * kBlk * 8) : 0;
    L.bp = o;    o += team ? al256((size_t)kBlk * 8) : 0;
    L.bv = o;    o += team ? al256((size_t)kBlk * 8) : 0;
    L.bmeta = o; o += team ? 256 : 0;
    L.total = o;
    return L;
}

// Rows each CTA of a team of G publishes (its best): G q <= kPubMax.
__host__ __device__ inline int cand_per_cta(int G) {
    int q = kPubMax / G;
    return q > 64 ? 64 : (q < 1 ? 1 : q);
}

// Dynamic shared memory of the blocked pass: the candidates (row, leverage),
// then the largest of its phases' work areas.
__host__ __device__ constexpr size_t block_smem() {
    constexpr size_t sort = (size_t)kSortMax * 16;
    constexpr size_t chol = (size_t)kCand * (kBlk + 1) * 8 + (size_t)kCand * (kCand + 1) / 2 * 8;
    constexpr size_t rows = (size_t)kBlk * kBlk * 8 + kBlk * 8 * 3 + (size_t)kSortMax * 9 +
                            (size_t)4 * 64 * (kBlk + 1) * 8;
    constexpr size_t w = sort > chol ? (sort > rows ? sort : rows) : (chol > rows ? chol : rows);
    return (size_t)kCand * 16 + w;
}

// Rows are processed TPR threads per row, THREADS / TPR rows at a time, so a
// CTA has many independent loads in flight (the products stream X from L2).
constexpr int kTPR = 8;

// sum_k x[k] * (CONJ ? conj(r[k]) : r[k]) over k < na, this thread's share:
// k-chunks sub, sub + TPR, ... of VEC = 16 / sizeof(S) elements (16-byte
// loads when VECTOR: x 16-byte aligned, r in shared memory), four chunks in
// flight, then the scalar tail.
template <typename S, bool VECTOR, bool CONJ>
__device__ __forceinline__ typename Tr<S>::A row_dot(const S *x, const S *r, int na, int sub) {
    using T = Tr<S>;
    using A = typename T::A;
    constexpr int V = VECTOR ? 16 / (int)sizeof(S) : 1;
    union Pack { uint4 u; S s[16 / sizeof(S)]; };
    A acc0 = T::zero(), acc1 = T::zero();
    int k = 0;
    if (VECTOR) {
        const int nv = na / V;
        int j = sub;
        for (; j + 3 * kTPR < nv; j += 4 * kTPR) {
            Pack a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u].u = *(const uint4 *)(x + (size_t)(j + u * kTPR) * V);
                b[u].u = *(const uint4 *)(r + (size_t)(j + u * kTPR) * V);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const A rv = CONJ ? T::conj(T::ld(&b[u].s[e])) : T::ld(&b[u].s[e]);
                    if (u & 1) acc1 = T::fma_(acc1, T::ld(&a[u].s[e]), rv);
                    else acc0 = T::fma_(acc0, T::ld(&a[u].s[e]), rv);
                }
        }
        for (; j < nv; j += kTPR) {
            Pack a, b;
            a.u = *(const uint4 *)(x + (size_t)j * V);
            b.u = *(const uint4 *)(r + (size_t)j * V);
#pragma unroll
            for (int e = 0; e < V; ++e)
                acc0 = T::fma_(acc0, T::ld(&a.s[e]), CONJ ? T::conj(T::ld(&b.s[e])) : T::ld(&b.s[e]));
        }
        k = nv * V;
    }
#pragma unroll 4
    for (int kk = k + sub; kk < na; kk += kTPR)
        acc1 = T::fma_(acc1, T::ld(x + kk), CONJ ? T::conj(T::ld(r + kk)) : T::ld(r + kk));
    return T::add(acc0, acc1);
}

// Sum over the kTPR consecutive lanes of a row group (all lanes take part).
template <typename A, typename T>
__device__ __forceinline__ A group_sum(A v) {
    for (int o = kTPR / 2; o; o >>= 1) {
        if constexpr (T::cplx) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        } else {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
    }
    return v;
}

// Order of the candidate rows: the larger leverage first, then the smaller
// row index (the reference's argmax takes the first of equal values).
__device__ __forceinline__ bool before(double va, int64_t ia, double vb, int64_t ib) {
    return va > vb || (va == vb && ia < ib);
}

// Four consecutive columns k..k+3 of a packed row in FP64, those past column
// a as zeros.  k is a multiple of 4 below a, so the vector loads are aligned
// and stay inside the row (x_stride); through L2, other CTAs write X.
template <typename S>
__device__ __forceinline__ void load4(const S *row, int k, int a, double (&v)[4]) {
    if constexpr (sizeof(S) == 4) {
        const float4 x = __ldcg((const float4 *)(row + k));
        v[0] = (double)x.x; v[1] = (double)x.y; v[2] = (double)x.z; v[3] = (double)x.w;
    } else {
        const double2 x = __ldcg((const double2 *)(row + k));
        double2 y = make_double2(0.0, 0.0);
        if (k + 2 < a) y = __ldcg((const double2 *)(row + k + 2));
        v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
    }
    if (k + 4 > a) {
#pragma unroll
        for (int e = 1; e < 4; ++e)
            if (k + e >= a) v[e] = 0.0;
    }
}

// One warp's share of the products of 8 RT rows of X with 8 CT rows over the
// first `a` columns, in FP64 on the matrix unit (m8n8k4): pa[r] is the row
// 8 r + lane / 4 of the first set, pb[c] of the second, and acc[r][c] holds
// the products of row lane / 4 of tile r with rows 2 (lane % 4) and
// 2 (lane % 4) + 1 of tile c.  A lane's four consecutive columns (one 16-byte load
// of FP32) feed four instructions, which permutes the columns of a 16-column
// step alike on both sides.  Steps share, share + shares, ... are this warp's.
// The operands go from L2 to registers: a CTA reads each row of its own set
// once, so staging through shared memory would only add a pass.
template <typename S, int RT, int CT>
__device__ __forceinline__ void warp_dots(const S *const (&pa)[RT], const S *const (&pb)[CT], int a, int share,
                                          int shares, double (&acc)[RT][CT][2]) {
    const int k1 = 4 * (threadIdx.x & 3);
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int c = 0; c < CT; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
#pragma unroll 2
    for (int k0 = 16 * share; k0 < a; k0 += 16 * shares) {
        const int k = k0 + k1;
        double x[RT][4], y[CT][4];
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[r][e] = 0.0;
#pragma unroll
        for (int c = 0; c < CT; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) y[c][e] = 0.0;
        if (k < a) {
#pragma unroll
            for (int r = 0; r < RT; ++r) load4(pa[r], k, a, x[r]);
#pragma unroll
            for (int c = 0; c < CT; ++c) load4(pb[c], k, a, y[c]);
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                 : "+d"(acc[r][c][0]), "+d"(acc[r][c][1])
                                 : "d"(x[r][e]), "d"(y[c][e]));
    }
}

// This CTA's best q rows by leverage ("before" order: bitonic sort of its
// nrow <= kSortMax rows in `work`), written to out[0..q).  own[i] is the leverage
// of row r0 + i.
__device__ void publish_best(const double *own, int64_t r0, int nrow, int q, Slot *out, unsigned char *work) {
    double *kv = (double *)work;
    int64_t *ki = (int64_t *)(work + (size_t)kSortMax * 8);
    const int tid = threadIdx.x;
    int np2 = 64;
    while (np2 < nrow || np2 < q) np2 <<= 1;
    for (int i = tid; i < np2; i += kThreads) {
        kv[i] = i < nrow ? own[i] : -1e300;
        ki[i] = i < nrow ? r0 + i : INT64_MAX;
    }
    __syncthreads();
    for (int k = 2; k <= np2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < np2; i += kThreads) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const bool up = (i & k) == 0;
                    const bool sw = up ? before(kv[ixj], ki[ixj], kv[i], ki[i]) : before(kv[i], ki[i], kv[ixj], ki[ixj]);
                    if (sw) {
                        const double tv = kv[i];
                        kv[i] = kv[ixj];
                        kv[ixj] = tv;
                        const int64_t ti = ki[i];
                        ki[i] = ki[ixj];
                        ki[ixj] = ti;
                    }
                }
            }
            __syncthreads();
        }
    for (int i = tid; i < q; i += kThreads) out[i] = {kv[i], ki[i]};
    __syncthreads();
}

// The same for q <= 16 of at most 256 rows, by one warp: eight rows a lane,
// the best taken q times by 32-bit reductions over the leverage's high word,
// low word and row (0.3 us for two of 64 rows, the sort 9 us).  `first` gets
// the best row (row 0 with the lowest value when no leverage is a number).
constexpr int kFewRows = 256, kFewBest = 16;
__device__ void publish_few(const double *own, int64_t r0, int nrow, int q, Slot *out, Slot *first) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int E = kFewRows / 32;
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    unsigned long long key[E];                             // ordered bits; 0: none
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = lane + 32 * e;
        const double v = i < nrow ? own[i] : -1e300;
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        key[e] = v > -1e300 ? ((long long)b < 0 ? ~b : b | (1ull << 63)) : 0ull;
    }
    for (int r = 0; r < q; ++r) {
        unsigned long long k = 0;
        int at = 0;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (key[e] > k) { k = key[e]; at = e; }        // first of equals: the smaller row
        const unsigned hi = (unsigned)(k >> 32), mh = __reduce_max_sync(FULL, hi);
        const unsigned lo = hi == mh ? (unsigned)k : 0u, ml = __reduce_max_sync(FULL, lo);
        const unsigned row = k && hi == mh && lo == ml ? (unsigned)(lane + 32 * at) : ~0u;
        const unsigned mr = __reduce_min_sync(FULL, row);
        const unsigned long long best = ((unsigned long long)mh << 32) | ml;
        const long long b = (long long)(best >> 63 ? best & ~(1ull << 63) : ~best);
        const bool any = mr != ~0u;
        if (lane == 0) {
            const double v = any ? __longlong_as_double(b) : -1e300;
            out[r] = {v, any ? r0 + (int64_t)mr : INT64_MAX};
            if (r == 0) *first = {v, any ? r0 + (int64_t)mr : 0};
        }
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (row == mr && at == e) key[e] = 0ull;
    }
}

// Blocked pass of the team path (real types).  The missing columns are the
// pivoted Cholesky factor of the projector P = I - X X^T onto the complement
// of the packed columns X, pivot = the largest leverage (P's remaining
// diagonal), exactly as the per-column loop builds them: column k =
// P_k e_p / sqrt(lev_p).  A block of up to kBlk columns is built
// speculatively on a candidate set C (the kCand best of every CTA's best
// rows), then checked:
//   P2  M = P[C, C] (diagonal: the tracked leverages; off-diagonal
//       -X_i . X_j in FP64), its lower triangle shared out over the team in
//       16 x 16 tiles, the columns over the warps of a CTA;
//   P3  CTA 0: the pivoted Cholesky of M, pivot = the best remaining
//       leverage in C, until kBlk columns, the missing columns run out, or
//       the best is below 1/2 (the per-column loop then takes that column,
//       with its second projection);
//   P4  every CTA forms its rows of the block, Y = E_S - X X_S^T and
//       N = Y L_SS^-T (forward substitution with the factor's pivot rows),
//       stores N as the next packed columns, and checks every row outside C
//       step by step: a row whose leverage at step s ranks before the
//       pivot's would have been step s's pivot, so the block keeps only the
//       steps before the first such s (step 0 always stands: the best row of
//       all is in C); the slots and the next block's candidates are
//       published as if all steps stood;
//   P5  when they do not: the leverages lowered by |N_i|^2 over the kept
//       steps, slots and candidates published again.
// The kept pivots and columns are, in exact arithmetic, the per-column
// loop's, at three team barriers per block instead of one per column.
// `fresh`: the candidate lists match the current leverages (else P1
// publishes them first).  Returns the columns completed (0: the per-column
// loop takes the next one), or -1 when a barrier wait ran out; `slow` is set
// when the block ended on a leverage below 1/2.
template <typename S>
__device__ int block_pass(const Params &p, const Layout &L, unsigned char *base, S *X, int64_t ldx, double *lev,
                          int a, const uint8_t *keep, int64_t c, int *cmap, Slot *slots, unsigned *bar,
                          unsigned char *smem, int G, int g, int64_t r0, int64_t r1, bool &fresh, bool &slow,
                          Slot *s_red) {
    using T = Tr<S>;
    constexpr unsigned FULL = 0xffffffffu;
    const int64_t n = p.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = cand_per_cta(G), npub = G * q, nc = npub < kCand ? npub : kCand;
    Slot *cand = (Slot *)(base + L.cand);
    double *bm = (double *)(base + L.bm);
    double *bl = (double *)(base + L.bl);
    int64_t *bp = (int64_t *)(base + L.bp);
    double *bpv = (double *)(base + L.bv);
    int *bmeta = (int *)(base + L.bmeta);
    int64_t *cidx = (int64_t *)smem;                       // candidates: row, leverage
    double *cval = (double *)(smem + kCand * 8);
    unsigned char *work = smem + kCand * 16;
    __shared__ int s_nmiss, s_fail;
    const int nrow = (int)(r1 - r0);
    slow = false;

    if (!fresh) {                                          // P1
        __shared__ Slot s_first;
        if (q <= kFewBest && nrow <= kFewRows) publish_few(lev + r0, r0, nrow, q, cand + (size_t)g * q, &s_first);
        else publish_best(lev + r0, r0, nrow, q, cand + (size_t)g * q, work);
        if (!team_sync(bar, G)) return -1;
    }
    fresh = false;
    // P2
    if (tid < kCand) {
        cidx[tid] = tid < npub ? __ldcg(&cand[tid].idx) : INT64_MAX;
        cval[tid] = tid < npub ? __ldcg(&cand[tid].val) : -1e300;
    }
    if (npub > kCand) {
        // The kCand best of the published rows, by their ranks: keys of the
        // leverage to 2^-44 and the place in the list, two threads a row.
        // (Any set will do that holds the best row: P4 checks the others.)
        unsigned long long *key = (unsigned long long *)work;
        const int t = tid >> 1, h = tid & 1;
        Slot mine = {-1e300, INT64_MAX};
        if (t < npub) mine = {__ldcg(&cand[t].val), __ldcg(&cand[t].idx)};
        const bool real = mine.idx != INT64_MAX && mine.val > 0.0;
        const unsigned long long kt =
            (real ? (unsigned long long)__double_as_longlong(mine.val) & ~255ull : 0ull) | (unsigned)(255 - t);
        if (h == 0) key[t] = kt;
        __syncthreads();
        int rank = 0;
        const ulonglong2 *kp = (const ulonglong2 *)key + 64 * h;
#pragma unroll 8
        for (int u = 0; u < 64; ++u) {
            const ulonglong2 k2 = kp[u];
            rank += (k2.x > kt) + (k2.y > kt);
        }
        rank += __shfl_xor_sync(FULL, rank, 1);
        if (h == 0 && rank < kCand) {
            cidx[rank] = mine.idx;
            cval[rank] = mine.val;
        }
    }
    __syncthreads();
    {
        constexpr int LDP = 17;
        double *part = (double *)work;                     // [warp][16][16] (ld LDP)
        const int nt = (nc + 15) / 16, tiles = nt * (nt + 1) / 2;
        for (int tt = g; tt < tiles; tt += G) {
            int ti = (int)((sqrtf(8.f * (float)tt + 1.f) - 1.f) * 0.5f);
            while (ti * (ti + 1) / 2 > tt) --ti;
            while ((ti + 1) * (ti + 2) / 2 <= tt) ++ti;
            const int i0 = 16 * ti, j0 = 16 * (tt - ti * (ti + 1) / 2);
            // padding and absent candidates read row 0; their products are not used
            const S *pa[2], *pb[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int64_t ra = cidx[i0 + 8 * r + (lane >> 2)], rb = cidx[j0 + 8 * r + (lane >> 2)];
                pa[r] = X + (ra != INT64_MAX ? ra : 0) * ldx;
                pb[r] = X + (rb != INT64_MAX ? rb : 0) * ldx;
            }
            double acc[2][2][2];
            warp_dots<S, 2, 2>(pa, pb, a, warp, kWarps, acc);
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        part[(warp * 16 + 8 * r + (lane >> 2)) * LDP + 8 * cc + 2 * (lane & 3) + e] = acc[r][cc][e];
            __syncthreads();
            if (tid < 256) {
                const int r = tid >> 4, cc = tid & 15, ia = i0 + r, jb = j0 + cc;
                double y = 0.0;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) y += part[(w * 16 + r) * LDP + cc];
                const bool ok = cidx[ia] != INT64_MAX && cidx[jb] != INT64_MAX;
                const double v = ok ? (ia == jb ? cval[ia] : -y) : 0.0;
                bm[ia * kCand + jb] = v;
            }
            __syncthreads();
        }
    }
    if (!team_sync(bar, G)) return -1;

    // P3: CTA 0, the pivoted Cholesky of M.  A serial chain of up to kBlk
    // steps, so the step is kept short: four threads a candidate with its row
    // of the factor in registers (every fourth step each), the pivot's row a
    // broadcast from shared memory, M's lower triangle staged there (the L2
    // latency of its row would be in every step), the best candidate by 32-bit
    // warp reductions over the leverage's high word, low word and row, and
    // one barrier.  One thread a candidate with the factor in shared memory
    // and M behind L2 took 59 us a block (8192 rows, 256 candidates); this form takes 22.
    // Two threads a candidate: 31 us, the factor's row and its select twice as
    // long and 1 / sqrt in the chain.
    if (g == 0) {
        constexpr int LDL = kBlk + 1;                      // odd: candidates' rows in different banks
        double *Lc = (double *)work;                       // L[t][s], kCand x kBlk (ld LDL)
        double *Mp = Lc + (size_t)kCand * LDL;             // lower triangle of M by rows
        __shared__ int s_pa[kBlk], s_cols[kBlk];           // candidate, U column of pivot s
        __shared__ double s_pv[kBlk];                      // leverage of pivot s
        __shared__ uint4 s_best[2][kWarps];                // leverage high, low, row, candidate
        constexpr int TP = 4, LE = kBlk / TP;              // threads a candidate, steps a thread
        const int t = tid / TP, h = tid % TP;
        const bool real = t < nc && cidx[t] != INT64_MAX;
        for (int i = tid; i < nc * LDL; i += kThreads) Lc[i] = 0.0;
        constexpr int RB = 4, CB = kCand / 32;             // rows of M in flight a warp, words a lane and row
        for (int i0 = warp; i0 < nc; i0 += RB * kWarps) {
            double v[RB][CB];
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int k = 0; k < CB; ++k) {
                    const int i = i0 + kWarps * r, kk = lane + 32 * k;
                    v[r][k] = i < nc && kk <= i ? __ldcg(bm + i * kCand + kk) : 0.0;
                }
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int k = 0; k < CB; ++k) {
                    const int i = i0 + kWarps * r, kk = lane + 32 * k;
                    if (i < nc && kk <= i) Mp[i * (i + 1) / 2 + kk] = v[r][k];
                }
        }
        if (warp == kWarps - 1) {
            int k = 0;
            for (int64_t c0 = c; c0 < n && k < kBlk; c0 += 32) {
                const bool miss = c0 + lane < n && !keep[c0 + lane];
                const unsigned bm_ = __ballot_sync(FULL, miss);
                const int at = k + __popc(bm_ & ((1u << lane) - 1u));
                if (miss && at < kBlk) s_cols[at] = (int)(c0 + lane);
                k += __popc(bm_);
            }
            if (lane == 0) s_nmiss = k < kBlk ? k : kBlk;
        }
        double d = real ? cval[t] : 0.0, l[LE];            // remaining leverage; steps TP j + h
#pragma unroll
        for (int j = 0; j < LE; ++j) l[j] = 0.0;
        bool open = real;                                  // a candidate that is no pivot yet
        const unsigned row = real ? (unsigned)cidx[t] : ~0u;
        // the lane with the best of the warp's (leverage bits, row) keys, "before"
        // order, or -1; one reduction unless high words tie
        auto best_lane = [&](unsigned hi, unsigned lo, unsigned rw, bool in) -> int {
            const unsigned mh = __reduce_max_sync(FULL, in ? hi : 0u);
            unsigned b = __ballot_sync(FULL, in && hi == mh);
            if (b & (b - 1u)) {
                const bool e0 = in && hi == mh;
                const unsigned ml = __reduce_max_sync(FULL, e0 ? lo : 0u);
                const unsigned mr = __reduce_min_sync(FULL, e0 && lo == ml ? rw : ~0u);
                b = __ballot_sync(FULL, e0 && lo == ml && rw == mr);
            }
            return __ffs(b) - 1;
        };
        // this warp's best open candidate (none above zero: key 0)
        auto warp_best = [&](int buf) {
            const int dh = __double2hiint(d);
            const unsigned hi = dh > 0 ? (unsigned)dh : 0u, lo = dh > 0 ? (unsigned)__double2loint(d) : 0u;
            const int w = best_lane(hi, lo, row, open && h == 0);
            if (w < 0 ? lane == 0 : lane == w) s_best[buf][warp] = make_uint4(hi, lo, row, w < 0 ? ~0u : (unsigned)t);
        };
        warp_best(0);
        __syncthreads();
        const int nmax = s_nmiss;
        int ns = 0, stop_slow = 0;
        for (; ns < nmax; ++ns) {
            const uint4 mine = s_best[ns & 1][lane & (kWarps - 1)];
            const int w = best_lane(mine.x, mine.y, mine.z, lane < kWarps && (int)mine.w >= 0);
            const uint4 top = s_best[ns & 1][w < 0 ? 0 : w];
            const int pb = w < 0 ? -1 : (int)top.w;
            if (pb < 0 || top.x < 0x3fe00000u) {           // none left, or its leverage below 1/2
                stop_slow = pb >= 0;
                break;
            }
            const double bv = __hiloint2double((int)top.x, (int)top.y);
            const double mt = open ? (t <= pb ? Mp[pb * (pb + 1) / 2 + t] : Mp[t * (t + 1) / 2 + pb]) : 0.0;
            // 1 / sqrt(bv), bv in [1/2, 2): FP32 estimate and one third-order
            // step (the residual e is 1e-7), beside the product's chain
            const double r0_ = (double)rsqrtf((float)bv);
            const double e_ = fma(-bv * r0_, r0_, 1.0);
            const double rp = fma(r0_ * e_, fma(0.375, e_, 0.5), r0_);
            const double *lp = Lc + pb * LDL + h;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
            for (int j = 0; j < LE; j += 4)
                if (TP * j < ns) {
                    s0 = fma(l[j], lp[TP * j], s0);
                    s1 = fma(l[j + 1], lp[TP * (j + 1)], s1);
                    s2 = fma(l[j + 2], lp[TP * (j + 2)], s2);
                    s3 = fma(l[j + 3], lp[TP * (j + 3)], s3);
                }
            double sum = (s0 + s1) + (s2 + s3);
            sum += __shfl_xor_sync(FULL, sum, 1);
            sum += __shfl_xor_sync(FULL, sum, 2);
            const double v = (mt - sum) * rp;
            open = open && t != pb;
            if (open) {
                d = fma(-v, v, d);
                if (h == 0) Lc[t * LDL + ns] = v;
            }
#pragma unroll
            for (int j = 0; j < LE; ++j) {
                int at = TP * j + h;
                asm("" : "+r"(at));                        // a select, not an indexed store to local memory
                l[j] = ns == at ? v : l[j];
            }
            warp_best((ns + 1) & 1);
            if (tid == 0) {
                s_pa[ns] = pb;
                s_pv[ns] = bv;
            }
            __syncthreads();                               // the factor's column and the warps' bests
        }
        for (int i = tid; i < ns * kBlk; i += kThreads) {
            const int r = i / kBlk, k = i - r * kBlk;
            bl[i] = k < r ? Lc[s_pa[r] * LDL + k] : (k == r ? sqrt(s_pv[r]) : 0.0);
        }
        for (int i = tid; i < ns; i += kThreads) {
            bp[i] = cidx[s_pa[i]];
            bpv[i] = s_pv[i];
            cmap[a + i] = s_cols[i];
        }
        if (tid == 0) {
            bmeta[0] = ns;
            bmeta[1] = stop_slow;
            bmeta[2] = ns;                                 // the first failing step (P4), at most ns
        }
    }
    if (!team_sync(bar, G)) return -1;
    const int ns = __ldcg(bmeta);
    if (ns == 0) {
        slow = __ldcg(bmeta + 1) != 0;
        fresh = true;                                      // the leverages did not change
        return 0;
    }

    // P4: this CTA's rows of the block, 64 at a time, and the check.  Warp w
    // forms the products of 16 rows with the pivots over a quarter of the
    // columns; then eight threads a row run the forward substitution, four
    // columns of the block each, the step's value a shuffle, and check the
    // leverages afterwards.
    constexpr int LDY = kBlk + 1;
    double *Lt = (double *)work;                           // kBlk x kBlk, Lt[s][t] = L[t][s] below the diagonal
    double *Li = Lt + kBlk * kBlk;                         // 1 / L[s][s]
    double *Pv = Li + kBlk;                                // pivot leverages
    int64_t *Sv = (int64_t *)(Pv + kBlk);                  // pivot rows
    double *lvs = (double *)(Sv + kBlk);                   // own rows' leverages after the whole block
    unsigned char *incand = (unsigned char *)(lvs + kSortMax);   // own rows in C
    double *part = (double *)(incand + kSortMax);          // [quarter][64][kBlk] (ld LDY); later the sort's area
    for (int i = tid; i < kBlk * kBlk; i += kThreads) {
        const int r = i / kBlk, k = i - r * kBlk;
        Lt[k * kBlk + r] = r < ns && k < r ? __ldcg(bl + i) : 0.0;
    }
    for (int i = tid; i < kBlk; i += kThreads) {
        Sv[i] = i < ns ? __ldcg(bp + i) : INT64_MAX;
        Pv[i] = i < ns ? __ldcg(bpv + i) : 0.0;
        Li[i] = i < ns ? 1.0 / __ldcg(bl + i * kBlk + i) : 0.0;
    }
    for (int i = tid; i < nrow; i += kThreads) incand[i] = 0;
    if (tid == 0) s_fail = ns;
    __syncthreads();
    for (int i = tid; i < nc; i += kThreads)
        if (cidx[i] >= r0 && cidx[i] < r1) incand[cidx[i] - r0] = 1;
    int fail = ns;
    for (int64_t rc = r0; rc < r1; rc += 64) {
        const int nr = (int)((r1 - rc) < 64 ? (r1 - rc) : 64);
        const int rg = warp & 3, kq = warp >> 2;
        if (16 * rg < nr) {
            const S *pa[2], *pb[4];                        // rows past the last, absent pivots: not used
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int i = 16 * rg + 8 * r + (lane >> 2);
                pa[r] = X + (rc + (i < nr ? i : 0)) * ldx;
            }
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const int64_t i = Sv[8 * cc + (lane >> 2)];
                pb[cc] = X + (i != INT64_MAX ? i : r0) * ldx;
            }
            double acc[2][4][2];
            warp_dots<S, 2, 4>(pa, pb, a, kq, 4, acc);
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        part[(kq * 64 + 16 * rg + 8 * r + (lane >> 2)) * LDY + 8 * cc + 2 * (lane & 3) + e] =
                            acc[r][cc][e];
        }
        __syncthreads();                                   // the products; incand in the first pass
        {
            const int rl = tid >> 3, sub = tid & 7;
            const bool own = rl < nr;
            const int64_t i = rc + (own ? rl : 0);
            const int il = (int)(i - r0);
            const bool check = own && !incand[il];
            double y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double *yp = part + (own ? rl : 0) * LDY + 4 * sub + e;
                y[e] = (i == Sv[4 * sub + e] ? 1.0 : 0.0) -
                       ((yp[0] + yp[64 * LDY]) + (yp[128 * LDY] + yp[192 * LDY]));
            }
            for (int s4 = 0; s4 < ns; s4 += 4) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {              // steps past ns: Li and Lt are zero
                    const double ys = __shfl_sync(FULL, y[e] * Li[s4 + e], s4 >> 2, 8);
                    const double2 *lt = (const double2 *)(Lt + (s4 + e) * kBlk + 4 * sub);
                    const double2 l0 = lt[0], l1 = lt[1];
                    y[0] = fma(-ys, l0.x, y[0]);
                    y[1] = fma(-ys, l0.y, y[1]);
                    y[2] = fma(-ys, l1.x, y[2]);
                    y[3] = fma(-ys, l1.y, y[3]);
                    if (sub == s4 >> 2) y[e] = ys;
                }
            }
            // the leverage before each of this thread's four steps: the squares
            // of the stored values, summed over the threads before it
            double sq[4], pre = 0.0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double st = 4 * sub + e < ns ? (double)(S)y[e] : 0.0;
                sq[e] = st * st;
                pre += sq[e];
            }
            double run = pre;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const double up = __shfl_up_sync(FULL, run, o, 8);
                if (sub >= o) run += up;
            }
            double lv = lev[i] - (run - pre);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int s2 = 4 * sub + e;
                if (check && s2 < fail && before(lv, i, Pv[s2], Sv[s2])) fail = s2;
                lv -= sq[e];
            }
            if (own) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * sub + e < ns) X[i * ldx + a + 4 * sub + e] = (S)y[e];
                if (sub == 7) lvs[il] = lv;
            }
        }
        __syncthreads();
    }
    if (fail < ns) atomicMin(&s_fail, fail);
    __syncthreads();
    // P5, as if every step of the block stands (the usual case): the slots
    // and the next block's candidates from the new leverages, before the
    // team agrees on the steps kept, so that one barrier serves both.
    auto publish = [&](const double *own) {
        if (q <= kFewBest && nrow <= kFewRows) {
            publish_few(own, r0, nrow, q, cand + (size_t)g * q, slots + g);
            return;
        }
        double best = -1e300;
        int64_t bidx = 0;
        for (int i = tid; i < nrow; i += kThreads)
            if (own[i] > best) { best = own[i]; bidx = r0 + i; }
        const Slot sb = cta_argmax(best, bidx, s_red);
        if (tid == 0) slots[g] = sb;
        publish_best(own, r0, nrow, q, cand + (size_t)g * q, (unsigned char *)part);
    };
    publish(lvs);
    if (tid == 0 && s_fail < ns) atomicMin(bmeta + 2, s_fail);
    if (!team_sync(bar, G)) return -1;
    const int kept = __ldcg(bmeta + 2);
    if (kept == ns) {
        for (int i = tid; i < nrow; i += kThreads) lev[r0 + i] = lvs[i];
        __syncthreads();
    } else {
        for (int64_t i = r0 + tid; i < r1; i += kThreads) {
            double lv = lev[i];
            const S *xi = X + i * ldx + a;
#pragma unroll 8
            for (int s2 = 0; s2 < kept; ++s2) {
                const double x = (double)__ldcg(xi + s2);
                lv -= x * x;
            }
            lev[i] = lv;
        }
        __syncthreads();
        publish(lev + r0);
        if (!team_sync(bar, G)) return -1;
    }
    fresh = true;
    slow = kept == ns && __ldcg(bmeta + 1) != 0;
    return kept;
}

// TEAM = false: one CTA per matrix, in place on U (the columns not yet
// completed are zero, so every product runs over all n columns, as the
// reference's u @ (u^H v) does; the new column is excluded from the second
// projection).  TEAM = true: a cooperative team of G CTAs, the kept and
// completed columns packed into X (row stride x_stride(n)), G > 1.
template <typename S, bool TEAM>
__global__ void __launch_bounds__(kThreads, 1) null_kernel(Params p) {
    using T = Tr<S>;
    using A = typename T::A;
    constexpr int kGroups = kThreads / kTPR;
    extern __shared__ __align__(16) unsigned char smem[];
    S *rowc = (S *)smem;                                   // row idx of X; y in the second projection
    __shared__ Slot s_red[kWarps];
    __shared__ double s_dred[kWarps];
    __shared__ int s_flag;
    __shared__ Slot s_piv;
    __shared__ double s_sum;
    const int G = TEAM ? p.G : 1;
    const int g = TEAM ? blockIdx.x : 0;                   // rank in the team
    const int64_t team = TEAM ? 0 : blockIdx.x;
    const int64_t nteams = TEAM ? 1 : gridDim.x;
    const int64_t m = p.m, n = p.n;
    const int64_t ldx = TEAM ? x_stride(n, sizeof(S)) : n;
    const Layout L = layout(m, n, sizeof(S), sizeof(A), G);
    unsigned char *base = p.ws + team * p.team_bytes;
    double *lev = (double *)(base + L.lev);
    A *y = (A *)(base + L.y);
    A *part = (A *)(base + L.part);
    int *cmap = (int *)(base + L.cmap);
    Slot *slots = (Slot *)(base + L.slots);                // [2][G]
    unsigned *bar = (unsigned *)(base + L.bar);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = threadIdx.x % kTPR, grp = threadIdx.x / kTPR;
    const int64_t r0 = m * g / G, r1 = m * (g + 1) / G;   // this CTA's rows
    // cross-CTA data is read through L2 (ld.global.cg): L1 is not coherent
    auto ldx_ = [&](const S *q) -> A { return TEAM ? T::ldcg(q) : T::ld(q); };
    auto ldy = [&](const A *q) -> A { return TEAM ? T::ldcgA(q) : *q; };
    int64_t z = team;
    for (; z < p.batch; z += nteams) {
        S *U = (S *)p.U + z * m * n;
        S *X = TEAM ? (S *)(base + L.x) : U;
        const uint8_t *keep = p.keep + z * n;
        if (warp == 0) {                                   // kept columns in order (cmap), by ballots
            int a = 0, miss = 0;
            for (int64_t c0 = 0; c0 < n; c0 += 32) {
                const int64_t c = c0 + lane;
                const bool in = c < n, kp = in && keep[c] != 0;
                const unsigned bk = __ballot_sync(0xffffffffu, kp);
                if (TEAM && kp) cmap[a + __popc(bk & ((1u << lane) - 1u))] = (int)c;
                a += __popc(bk);
                miss += __popc(__ballot_sync(0xffffffffu, in && !kp));
            }
            if (lane == 0) s_flag = miss ? a : -1;
        }
        __syncthreads();
        const int nkept = s_flag;
        if (nkept < 0) {                                   // nothing to complete
            if (g == 0 && threadIdx.x == 0) p.status[z] = JB_ST_OK;
            __syncthreads();                               // s_flag is rewritten for the next matrix
            continue;
        }
        // Zero U's missing columns (primitives.py:436), pack the kept ones
        // (TEAM), leverage of every row of this CTA in FP64.
        double best = -1e300;
        int64_t bidx = 0;
        for (int64_t i = r0 + warp; i < r1; i += kWarps) {
            S *urow = U + i * n;
            double acc = 0.0;
            for (int64_t c = lane; c < n; c += 32) {
                if (!keep[c]) T::st(urow + c, T::zero());
                else acc += T::norm2(T::ld(urow + c));
            }
            if (TEAM)
                for (int k = lane; k < nkept; k += 32) X[i * ldx + k] = urow[cmap[k]];
            for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            const double lv = 1.0 - acc;
            if (lane == 0) lev[i] = lv;
            if (lv > best) { best = lv; bidx = i; }         // lanes agree; rows ascend
        }
        Slot sb = cta_argmax(best, bidx, s_red);
        if (threadIdx.x == 0) slots[g] = sb;
        if (!team_sync(bar, G)) goto timeout;
        {
            int a = nkept;                                 // packed columns (TEAM)
            bool failed = false;
            bool blocked = TEAM && !T::cplx && p.blocked;  // block_pass while it applies
            bool fresh = false;                            // its candidate lists are current
            for (int64_t c = 0; c < n; ++c) {
                if (keep[c]) continue;
                if constexpr (TEAM && !T::cplx) {
                    if (blocked) {
                        bool slow = false;
                        const int done = block_pass<S>(p, L, base, X, ldx, lev, a, keep, c, cmap, slots, bar, smem, G,
                                                       g, r0, r1, fresh, slow, s_red);
                        if (done < 0) goto timeout;
                        if (slow) blocked = false;
                        if (done > 0) {
                            a += done;
                            c = __ldcg(&cmap[a - 1]);              // the last column of the block
                            continue;
                        }
                    }
                    fresh = false;                         // the per-column step changes the leverages
                }
                const int na = TEAM ? a : (int)n;          // columns a product runs over
                const int64_t col = TEAM ? a : c;          // where v is built
                // idx = team-wide first argmax of the leverage
                const Slot piv = team_argmax(slots, G, TEAM, &s_piv);
                const int64_t idx = piv.idx;
                // The first projection's length^2 is the pivot's leverage (v = P e_idx
                // with P the projector onto the complement, so |v|^2 = P_idx,idx).  A
                // team that needs no second projection (leverage >= 1/2) normalises
                // by it at once and saves the team-wide norm reduction.
                const bool fast = TEAM && piv.val >= 0.5;
                const double inv_fast = fast ? 1.0 / sqrt(piv.val) : 0.0;
                for (int k = threadIdx.x; k < na; k += kThreads) T::st(rowc + k, ldx_(X + idx * ldx + k));
                __syncthreads();
                // first projection, row-local: v_i = delta - X_i . conj(X_idx)
                // (column col of X is still zero in every row)
                double pn2 = 0.0;
                best = -1e300;
                bidx = 0;
                for (int64_t i0 = r0; i0 < r1; i0 += kGroups) {
                    const int64_t i = i0 + grp;
                    A acc = i < r1 ? row_dot<S, TEAM, true>(X + i * ldx, rowc, na, sub) : T::zero();
                    acc = group_sum<A, T>(acc);
                    if (sub == 0 && i < r1) {
                        const A v = T::sub(i == idx ? T::unit() : T::zero(), acc);
                        if (fast) {
                            T::st(X + i * ldx + col, T::scale(v, inv_fast));
                            const double lv = lev[i] - T::norm2(T::ld(X + i * ldx + col));
                            lev[i] = lv;
                            if (lv > best) { best = lv; bidx = i; }
                        } else {
                            T::st(X + i * ldx + col, v);
                            pn2 += T::norm2(T::ld(X + i * ldx + col));
                        }
                    }
                }
                if (fast) {
                    sb = cta_argmax(best, bidx, s_red);
                    if (threadIdx.x == 0) {
                        slots[g] = sb;
                        if (g == 0) cmap[a] = (int)c;
                    }
                    ++a;
                    if (!team_sync(bar, G)) goto timeout;
                    continue;
                }
                double n2 = cta_sum(pn2, s_dred);
                if (threadIdx.x == 0) slots[G + g].val = n2;
                if (!team_sync(bar, G)) goto timeout;
                n2 = team_sum(slots + G, G, TEAM, &s_sum);
                if (p.always_reorth || n2 < 0.5) {
                    // second projection: y = X^H v (without v's own column), v -= X y
                    A *yout = TEAM ? part + (size_t)g * n : y;
                    for (int k = threadIdx.x; k < na; k += kThreads) {
                        A acc0 = T::zero(), acc1 = T::zero();
                        if (k != col) {
                            int64_t i = r0;
                            for (; i + 1 < r1; i += 2) {
                                acc0 = T::fma_(acc0, T::conj(T::ld(X + i * ldx + k)), T::ld(X + i * ldx + col));
                                acc1 = T::fma_(acc1, T::conj(T::ld(X + (i + 1) * ldx + k)),
                                               T::ld(X + (i + 1) * ldx + col));
                            }
                            if (i < r1) acc0 = T::fma_(acc0, T::conj(T::ld(X + i * ldx + k)), T::ld(X + i * ldx + col));
                        }
                        yout[k] = T::add(acc0, acc1);
                    }
                    if (TEAM) {
                        // every CTA sums the partials of its slice of y
                        if (!team_sync(bar, G)) goto timeout;
                        const int64_t k0 = (int64_t)na * g / G, k1 = (int64_t)na * (g + 1) / G;
                        for (int64_t k = k0 + threadIdx.x; k < k1; k += kThreads) {
                            A acc = T::zero();
                            for (int q = 0; q < G; ++q) acc = T::add(acc, T::ldcgA(part + (size_t)q * n + k));
                            y[k] = acc;
                        }
                    }
                    if (!team_sync(bar, G)) goto timeout;
                    // y in the input precision, as the reference's product (rowc is free again)
                    for (int k = threadIdx.x; k < na; k += kThreads) T::st(rowc + k, ldy(y + k));
                    __syncthreads();
                    double pn2b = 0.0;
                    for (int64_t i0 = r0; i0 < r1; i0 += kGroups) {
                        const int64_t i = i0 + grp;
                        A acc = i < r1 ? row_dot<S, TEAM, false>(X + i * ldx, rowc, na, sub) : T::zero();
                        acc = group_sum<A, T>(acc);
                        if (sub == 0 && i < r1) {
                            T::st(X + i * ldx + col, T::sub(T::ld(X + i * ldx + col), acc));
                            pn2b += T::norm2(T::ld(X + i * ldx + col));
                        }
                    }
                    const double s2 = cta_sum(pn2b, s_dred);
                    if (threadIdx.x == 0) slots[G + g].val = s2;
                    if (!team_sync(bar, G)) goto timeout;
                    n2 = team_sum(slots + G, G, TEAM, &s_sum);
                }
                const double len = sqrt(n2);
                if (len < 10.0 * T::eps) {                 // primitives.py:451-452
                    failed = true;
                    break;
                }
                // normalise, lower the leverage, next argmax
                const double inv = 1.0 / len;
                best = -1e300;
                bidx = 0;
                for (int64_t i = r0 + threadIdx.x; i < r1; i += kThreads) {
                    T::st(X + i * ldx + col, T::scale(T::ld(X + i * ldx + col), inv));
                    const double lv = lev[i] - T::norm2(T::ld(X + i * ldx + col));
                    lev[i] = lv;
                    if (lv > best) { best = lv; bidx = i; }
                }
                sb = cta_argmax(best, bidx, s_red);
                if (threadIdx.x == 0) {
                    slots[g] = sb;
                    if (TEAM && g == 0) cmap[a] = (int)c;
                }
                ++a;
                if (!team_sync(bar, G)) goto timeout;
            }
            if (TEAM)                                      // completed columns back into U
                for (int64_t i = r0 + warp; i < r1; i += kWarps)
                    for (int k = nkept + lane; k < a; k += 32) U[i * n + __ldcg(&cmap[k])] = X[i * ldx + k];
            if (g == 0 && threadIdx.x == 0) p.status[z] = failed ? JB_ST_NULL_FAILED : JB_ST_OK;
            if (!team_sync(bar, G)) goto timeout;
        }
    }
    return;
timeout:
    // a barrier wait ran out: this matrix and the team's later ones fail
    if (threadIdx.x == 0 && g == 0)
        for (; z < p.batch; z += nteams) p.status[z] = JB_ST_TIMEOUT;
}

struct Plan {
    int G, blocked;
    int64_t grid;
    size_t team_bytes, bytes, smem;
};

static int esize(int dtype) { return dtype == 0 ? 4 : dtype == 1 ? 8 : dtype == 2 ? 8 : 16; }

static int dev_sms() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return 148;
    return sms;
}

// One CTA per matrix unless the batch has few large matrices: then one
// cooperative team of up to one CTA per SM (about 64 rows each).
static Plan make_plan(int dtype, int64_t batch, int64_t m, int64_t n) {
    Plan pl;
    const int sms = dev_sms();
    const int esz = esize(dtype), asz = dtype >= 2 ? 16 : 8;
    const bool large = batch * 4 < sms && m * n >= (1 << 16) && m >= 256;
    pl.blocked = 0;
    if (large) {
        int64_t G = m / 64;                         // about 64 rows per CTA
        if (G > sms) G = sms;
        if (G < 2) G = 2;
        pl.G = (int)G;
        pl.grid = G;
        pl.team_bytes = layout(m, n, esz, asz, pl.G).total;
        pl.bytes = pl.team_bytes;
        // real types, at most kSortMax rows per CTA: the blocked pass
        pl.blocked = dtype <= 1 && (m + G - 1) / G <= kSortMax;
    } else {
        pl.G = 1;
        int64_t grid = (int64_t)sms * 4;
        if (grid > batch) grid = batch;
        if (grid < 1) grid = 1;
        pl.grid = grid;
        pl.team_bytes = layout(m, n, esz, asz, 1).total;
        pl.bytes = pl.team_bytes * (size_t)grid;
    }
    pl.smem = (size_t)n * esz;
    if (pl.blocked && pl.smem < block_smem()) pl.smem = block_smem();
    return pl;
}

template <typename S>
static int launch(Params &p, const Plan &pl, cudaStream_t st) {
    p.G = pl.G;
    p.team_bytes = pl.team_bytes;
    p.always_reorth = pl.G == 1;
    p.blocked = pl.blocked;
    if (pl.G == 1) {
        auto kern = null_kernel<S, false>;
        if (pl.smem > 48 * 1024 &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem) != cudaSuccess)
            return JB_ECUDA;
        kern<<<(unsigned)pl.grid, kThreads, pl.smem, st>>>(p);
        return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
    }
    auto kern = null_kernel<S, true>;
    if (pl.smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem) != cudaSuccess)
        return JB_ECUDA;
    // the barrier words and the error flag start at zero
    const Layout L = layout(p.m, p.n, sizeof(S), Tr<S>::cplx ? 16 : 8, pl.G);
    if (cudaMemsetAsync(p.ws + L.bar, 0, 256, st) != cudaSuccess) return JB_ECUDA;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, pl.smem) != cudaSuccess)
        return JB_ECUDA;
    if ((int64_t)per_sm * dev_sms() < pl.grid) return JB_ETOOBIG;   // every CTA must be resident
    void *args[] = {&p};
    if (cudaLaunchCooperativeKernel((const void *)kern, dim3((unsigned)pl.grid), dim3(kThreads), args, pl.smem,
                                    st) != cudaSuccess)
        return JB_ECUDA;
    return JB_OK;
}

}  // namespace nul
}  // namespace jb

using namespace jb::nul;

extern "C" {

size_t jb_complete_null_workspace_bytes(int32_t dtype, int64_t batch, int64_t m, int64_t n) {
    if (dtype < 0 || dtype > 3 || batch < 0 || m < 1 || n < 1) return 0;
    return make_plan(dtype, batch, m, n).bytes;
}

int jb_complete_null(void *U, const uint8_t *keep, int32_t dtype, int64_t batch, int64_t m, int64_t n,
                     int32_t *status, void *workspace, size_t workspace_bytes, void *stream) {
    if (!U || !keep || !status || dtype < 0 || dtype > 3 || batch < 0 || m < 1 || n < 1) return JB_EINVAL;
    if (n > 8192 || m > ((int64_t)1 << 31) / n) return JB_ETOOBIG;
    if (batch == 0) return JB_OK;
    const Plan pl = make_plan(dtype, batch, m, n);
    if (pl.smem > 227 * 1024) return JB_ETOOBIG;
    if (!workspace || workspace_bytes < pl.bytes) return JB_EWORKSPACE;
    Params p;
    p.U = U;
    p.keep = keep;
    p.status = status;
    p.batch = batch;
    p.m = m;
    p.n = n;
    p.ws = (unsigned char *)workspace;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case 0: return launch<float>(p, pl, st);
        case 1: return launch<double>(p, pl, st);
        case 2: return launch<cf>(p, pl, st);
        default: return launch<cd>(p, pl, st);
    }
}

}  // extern "C"
