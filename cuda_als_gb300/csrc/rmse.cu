// rmse.cu — squared error of a rating set against the factors, summed in FP64 in a fixed order.
//
// Replaces calculate_square_error + rsme_test/rsme_train (als_model.cu:62-89, 1722-1764): the
// reference adds FP32 squares into 1000 buckets with atomicAdd (non-deterministic order) and
// sums them with cublasSasum.  Here each thread accumulates its ratings in FP64, CTAs reduce in
// a fixed tree, and one CTA adds the CTA partials in index order, so the result is bit-for-bit
// repeatable.  The dot product keeps the reference's NaN rule: it stops at the first factor
// component that is NaN (als_model.cu:78-79).  Bound by the FP64 pipe (two lanes an SM and clock):
// one FMA per factor pair is what the FP64 sum needs, so the factors are widened by integer
// operations on their bits, which run beside it, instead of two conversions on that same pipe.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "internal.h"

namespace als {

namespace {

constexpr int RMSE_THREADS = 256;
constexpr int RMSE_BLOCKS = 152 * 8;  // fixed grid: the summation order never depends on size

__device__ double block_sum_d(double v, double *sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < RMSE_THREADS / 32; ++w) s += sh[w];
    return s;  // valid in thread 0
}

// (double)x for a normal x: the exponent rebiased by 1023 - 127, the fraction moved up 29 bits.
__device__ __forceinline__ double widen(uint32_t x) {
    const uint32_t hi = ((x & 0x7fffffffu) >> 3) + 0x38000000u;
    return __hiloint2double((int)(hi | (x & 0x80000000u)), (int)(x << 29));
}
// Whether x is zero, subnormal, infinite or NaN.
__device__ __forceinline__ bool special(uint32_t x) {
    return (x & 0x7fffffffu) - 0x00800000u >= 0x7f000000u;
}

// pred += sum of N factor pairs in order, one FP64 FMA each; false at a NaN component.
template <int N>
__device__ __forceinline__ bool add_pairs(const uint32_t (&a)[N], const uint32_t (&b)[N], double &pred) {
    bool plain = true;
#pragma unroll
    for (int k = 0; k < N; ++k) plain = plain && !special(a[k]) && !special(b[k]);
    if (plain) {
#pragma unroll
        for (int k = 0; k < N; ++k) pred = fma(widen(a[k]), widen(b[k]), pred);
        return true;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float x = __uint_as_float(a[k]), y = __uint_as_float(b[k]);
        if (x != x || y != y) return false;
        pred = fma((double)x, (double)y, pred);
    }
    return true;
}

// N: factors a load (N divides f, so every row starts on a load's boundary).  Measured at 1,408,395
// ratings, f = 100, N = 4: 816 us with conversions and scalar loads, now
// 280 us of which 240 are the FP64 FMAs (odd f: N = 1).
template <int N>
__global__ void __launch_bounds__(RMSE_THREADS)
sq_error_partials_kernel(int64_t nnz, const int32_t *__restrict__ rows,
                         const int32_t *__restrict__ cols, const float *__restrict__ vals,
                         const float *__restrict__ U, const float *__restrict__ V, int f,
                         double *__restrict__ partials) {
    __shared__ double sh[RMSE_THREADS / 32];
    double acc = 0.0;
    for (int64_t e = (int64_t)blockIdx.x * RMSE_THREADS + threadIdx.x; e < nnz;
         e += (int64_t)RMSE_BLOCKS * RMSE_THREADS) {
        const uint32_t *u = reinterpret_cast<const uint32_t *>(U + (int64_t)rows[e] * f);
        const uint32_t *v = reinterpret_cast<const uint32_t *>(V + (int64_t)cols[e] * f);
        double pred = 0.0;
        for (int i = 0; i < f; i += N) {
            uint32_t a[N], b[N];
            if constexpr (N == 4) {
                const uint4 x = __ldg(reinterpret_cast<const uint4 *>(u + i));
                const uint4 y = __ldg(reinterpret_cast<const uint4 *>(v + i));
                a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
                b[0] = y.x; b[1] = y.y; b[2] = y.z; b[3] = y.w;
            } else if constexpr (N == 2) {
                const uint2 x = __ldg(reinterpret_cast<const uint2 *>(u + i));
                const uint2 y = __ldg(reinterpret_cast<const uint2 *>(v + i));
                a[0] = x.x; a[1] = x.y;
                b[0] = y.x; b[1] = y.y;
            } else {
                a[0] = __ldg(u + i);
                b[0] = __ldg(v + i);
            }
            if (!add_pairs<N>(a, b, pred)) break;
        }
        const double err = (double)vals[e] - pred;
        acc = fma(err, err, acc);
    }
    double s = block_sum_d(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

__global__ void __launch_bounds__(RMSE_THREADS)
sum_partials_kernel(const double *__restrict__ partials, int n, double *__restrict__ out) {
    __shared__ double sh[RMSE_THREADS / 32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += RMSE_THREADS) acc += partials[i];
    double s = block_sum_d(acc, sh);
    if (threadIdx.x == 0) *out = s;
}

}  // namespace

size_t rmse_scratch_bytes() { return sizeof(double) * (RMSE_BLOCKS + 32); }

cudaError_t launch_sq_error(int64_t nnz, const int32_t *rows, const int32_t *cols,
                            const float *vals, const float *U, const float *V, int f,
                            double *d_partials, double *d_out, cudaStream_t st) {
    const auto kernel = (f & 3) == 0   ? sq_error_partials_kernel<4>
                        : (f & 1) == 0 ? sq_error_partials_kernel<2>
                                       : sq_error_partials_kernel<1>;
    kernel<<<RMSE_BLOCKS, RMSE_THREADS, 0, st>>>(nnz, rows, cols, vals, U, V, f, d_partials);
    sum_partials_kernel<<<1, RMSE_THREADS, 0, st>>>(d_partials, RMSE_BLOCKS, d_out);
    return cudaGetLastError();
}

// Relative difference of two factor tables over the rows order[lo..hi): sum (a - b)^2 and
// sum a^2 in FP64 (the autotuner's agreement check between two solvers).
static __global__ void bucket_diff_kernel(const int32_t *__restrict__ order, int32_t lo, int32_t hi,
                                   const float *__restrict__ A, const float *__restrict__ Bm, int f,
                                   double *__restrict__ out) {
    __shared__ double sd[32], sa[32];
    double d2 = 0.0, a2 = 0.0;
    const int64_t total = (int64_t)(hi - lo) * f;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = order[lo + e / f];
        const int j = (int)(e % f);
        const double a = A[r * f + j], b = Bm[r * f + j];
        d2 += (a - b) * (a - b);
        a2 += a * a;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        d2 += __shfl_xor_sync(0xffffffffu, d2, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sd[threadIdx.x >> 5] = d2;
        sa[threadIdx.x >> 5] = a2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double td = 0.0, ta = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            td += sd[w];
            ta += sa[w];
        }
        atomicAdd(&out[0], td);
        atomicAdd(&out[1], ta);
    }
}

cudaError_t launch_bucket_diff(const int32_t *order, int32_t lo, int32_t hi, const float *A,
                               const float *B, int f, double *out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, 2 * sizeof(double), st);
    if (e != cudaSuccess || hi <= lo) return e;
    const int64_t total = (int64_t)(hi - lo) * f;
    const int grid = (int)std::min<int64_t>((total + 255) / 256, 1216);
    bucket_diff_kernel<<<grid, 256, 0, st>>>(order, lo, hi, A, B, f, out);
    return cudaGetLastError();
}

}  // namespace als
