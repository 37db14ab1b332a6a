// jb_prep.cu - what svd() does around the solvers that are composed on the host:
// the finiteness check, the exact power-of-two scaling and the wide -> tall
// transposition of a batch before (svdbench/standalone/solvers.py:291-295,
// 224-227), the finiteness check of the outputs after (:305-306).
//
// Two launches a batch instead of about ten elementwise ones, and the verdicts
// stay on the device: the host reads them with the solver's status words in
// one copy, where it waited for every check.  Latency-bound (microseconds at
// these sizes); DRAM-bound beyond.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include "jacobi_b200.h"

namespace jb {
namespace prep {

constexpr int kThreads = 256;
constexpr int kPer = 16;   // elements a thread and block of the scan

// Exponent field of a positive finite double (at least 1), 0 of zero, 0x7ff of inf and NaN.
__device__ __forceinline__ int key_of(double a) {
    const int ex = (__double2hiint(a) >> 20) & 0x7ff;
    return a == 0.0 ? 0 : (ex > 1 ? ex : 1);
}
// amax = f 2^e with f in [0.5, 1) (e <= 1023, so that 2^e is finite); 0 for a zero or non-finite matrix
__device__ __forceinline__ int exponent_of(int key) {
    if (key == 0 || key == 0x7ff) return 0;
    return key - 1022 < 1023 ? key - 1022 : 1023;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) scan_kernel(const T *x, int32_t *keys, int64_t per_matrix) {
    const T *a = x + blockIdx.y * per_matrix;
    int key = 0;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < per_matrix; i += (int64_t)gridDim.x * kThreads) {
        const int k = key_of(fabs((double)a[i]));
        if (k > key) key = k;
    }
    key = __reduce_max_sync(0xffffffffu, key);
    if ((threadIdx.x & 31) == 0 && key) atomicMax(keys + blockIdx.y, key);
}

// NC reals an element; rows x cols per matrix.  TR: the (conjugate) transpose
// in 32 x 32 tiles through shared memory, else element by element.
template <typename T, typename TO, int NC, bool TR>
__global__ void __launch_bounds__(kThreads) scale_kernel(const T *x, TO *out, const int32_t *keys, double *scale,
                                                         int32_t *status, int rows, int cols) {
    const int64_t z = blockIdx.y, per = (int64_t)rows * cols;
    const int key = keys[z], e = exponent_of(key);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scale[z] = ldexp(1.0, e);
        status[z] = key == 0x7ff ? JB_ST_NONFINITE_IN : JB_ST_OK;
    }
    const T *a = x + z * per * NC;
    TO *o = out + z * per * NC;
    if constexpr (!TR) {
        for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < per * NC; i += (int64_t)gridDim.x * kThreads)
            o[i] = (TO)ldexp((double)a[i], -e);
    } else {
        __shared__ TO tile[32][32 * NC + 1];
        const int tc = (cols + 31) >> 5, tiles = ((rows + 31) >> 5) * tc;
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int r0 = (t / tc) << 5, c0 = (t % tc) << 5;
            for (int r = ty; r < 32; r += kThreads / 32)
                if (r0 + r < rows && c0 + tx < cols) {
                    const T *s = a + ((int64_t)(r0 + r) * cols + c0 + tx) * NC;
                    tile[r][NC * tx] = (TO)ldexp((double)s[0], -e);
                    if (NC == 2) tile[r][NC * tx + NC - 1] = (TO)ldexp(-(double)s[NC - 1], -e);
                }
            __syncthreads();
            for (int c = ty; c < 32; c += kThreads / 32)
                if (c0 + c < cols && r0 + tx < rows) {
                    TO *d = o + ((int64_t)(c0 + c) * rows + r0 + tx) * NC;
                    d[0] = tile[tx][NC * c];
                    if (NC == 2) d[NC - 1] = tile[tx][NC * c + NC - 1];
                }
            __syncthreads();
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) finite_kernel(const T *x, int32_t *flag, int64_t count) {
    int bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += (int64_t)gridDim.x * kThreads)
        if (!isfinite(x[i])) bad = 1;
    if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 1;
}

static unsigned blocks_for(int64_t count, int64_t most) {
    int64_t b = (count + kThreads * kPer - 1) / (kThreads * kPer);
    if (b > most) b = most;
    return (unsigned)(b < 1 ? 1 : b);
}

template <typename T, typename TO, int NC>
static int prepare(const T *x, TO *out, int transpose, double *scale, int32_t *keys, int32_t *status, int64_t batch,
                   int rows, int cols, cudaStream_t st) {
    const int64_t per = (int64_t)rows * cols;
    // the second grid dimension is limited to 65535 matrices a launch
    for (int64_t z = 0; z < batch; z += 65535) {
        const unsigned b = (unsigned)(batch - z < 65535 ? batch - z : 65535);
        const unsigned bx = blocks_for(per * NC, 1 + 4096 / b);
        scan_kernel<T><<<dim3(bx, b), kThreads, 0, st>>>(x + z * per * NC, keys + z, per * NC);
        if (transpose)
            scale_kernel<T, TO, NC, true><<<dim3(bx, b), kThreads, 0, st>>>(x + z * per * NC, out + z * per * NC, keys + z,
                                                                           scale + z, status + z, rows, cols);
        else
            scale_kernel<T, TO, NC, false><<<dim3(bx, b), kThreads, 0, st>>>(x + z * per * NC, out + z * per * NC, keys + z,
                                                                            scale + z, status + z, rows, cols);
    }
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

}  // namespace prep
}  // namespace jb

extern "C" {

int jb_prepare(const void *x, int32_t dtype, void *out, int32_t widen, int32_t transpose, double *scale, int32_t *keys,
               int32_t *status, int64_t batch, int32_t rows, int32_t cols, void *stream) {
    if (!x || !out || !scale || !keys || !status || batch < 0 || rows < 1 || cols < 1 || dtype < 0 || dtype > 3 ||
        (widen && dtype != 0))
        return JB_EINVAL;
    if (batch == 0) return JB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(keys, 0, (size_t)batch * 4, st) != cudaSuccess) return JB_ECUDA;
    using namespace jb::prep;
    if (widen) return prepare<float, double, 1>((const float *)x, (double *)out, transpose, scale, keys, status, batch, rows, cols, st);
    if (dtype == 0) return prepare<float, float, 1>((const float *)x, (float *)out, transpose, scale, keys, status, batch, rows, cols, st);
    if (dtype == 1) return prepare<double, double, 1>((const double *)x, (double *)out, transpose, scale, keys, status, batch, rows, cols, st);
    if (dtype == 2) return prepare<float, float, 2>((const float *)x, (float *)out, transpose, scale, keys, status, batch, rows, cols, st);
    return prepare<double, double, 2>((const double *)x, (double *)out, transpose, scale, keys, status, batch, rows, cols, st);
}

int jb_check_finite(const void *x, int32_t dtype, int64_t count, int32_t *flag, void *stream) {
    if (!x || !flag || count < 0 || dtype < 0 || dtype > 3) return JB_EINVAL;
    if (count == 0) return JB_OK;
    const int64_t reals = dtype >= 2 ? 2 * count : count;
    const unsigned b = jb::prep::blocks_for(reals, 2048);
    if (dtype & 1) jb::prep::finite_kernel<double><<<b, jb::prep::kThreads, 0, (cudaStream_t)stream>>>((const double *)x, flag, reals);
    else jb::prep::finite_kernel<float><<<b, jb::prep::kThreads, 0, (cudaStream_t)stream>>>((const float *)x, flag, reals);
    return cudaGetLastError() == cudaSuccess ? JB_OK : JB_ECUDA;
}

}  // extern "C"
