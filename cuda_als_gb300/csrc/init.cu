// init.cu — the reference's factor initialisation on the GPU, bit for bit.
//
// als_model::train starts from srand(0); VT[k] = 0.2 * ((float)rand() / (float)RAND_MAX) for
// k < n f, UT = 0 (als_model.cu:1772-1784).  glibc's rand() (the additive feedback generator of
// random_r, TYPE_3: degree 31, separation 3) is the linear recurrence
//   r_0 = seed (0 taken as 1), r_i = 16807 r_{i-1} mod (2^31 - 1) for 0 < i < 31,
//   r_i = r_{i-31} for 31 <= i < 34,  r_i = r_{i-31} + r_{i-3} (mod 2^32) for i >= 34,
// and the k-th call returns r_{344+k} >> 1.  With x the shift by one, x^31 = x^28 + 1 on the
// sequence, over Z/2^32:
//   * a jump by N is x^N reduced to 31 coefficients c_j: r_{i+N} = sum_j c_j r_{i+j};
//   * x^(31 m) = (x^28 + 1)^m: r_i = sum_k C(m, k) r_{i - 31 m + 28 k}, in which the nearest term
//     is 3 m back, so 3 m values follow from known ones at once.
// A warp makes WARP_CALLS calls: lane t jumps value t of the sequence's first 31 to the warp's
// place (one jump per set bit of its number, by constants worked out at compile time), then the
// warp grows the stretch with m = 1, 2, 4, 8.  Every output goes through the reference's own
// arithmetic: (float)(r >> 1) / (float)RAND_MAX in FP32 (RAND_MAX rounds to 2^31), times 0.2 in
// FP64, rounded to FP32.
// A chain of small dependent steps sets the time, so the stretches are short.  Against
// stretches of 1,984 calls a thread by 31 x 31 matrices that the host multiplied and uploaded:
// a training call of 5,000 values 1.39 -> 0.85 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace als {

namespace {

constexpr int DEG = 31;                     // the generator's degree
constexpr int WARP_CALLS = DEG * 32;        // rand() calls a warp makes: x^992 = x^31 squared five times
constexpr int STRETCH = DEG + WARP_CALLS;   // with the 31 values before them
constexpr int WINDOW = 2 * DEG - 1;         // what a jump of 31 values reads
constexpr int WARPS = 4;
constexpr int MAX_JUMPS = 36;               // jumps by 2^k stretches: n f < 2^45

struct Tables {
    uint32_t start[WINDOW];            // r_313 .. r_373: the 31 values before call 0, and 30 more
    uint32_t jump[MAX_JUMPS][DEG];     // x^(WARP_CALLS 2^k)
};

constexpr void square(uint32_t (&c)[DEG]) {
    uint32_t p[2 * DEG - 1] = {};
    for (int i = 0; i < DEG; ++i)
        for (int j = 0; j < DEG; ++j) p[i + j] += c[i] * c[j];
    for (int d = 2 * DEG - 2; d >= DEG; --d) {  // x^d = x^(d - 3) + x^(d - 31)
        p[d - 3] += p[d];
        p[d - DEG] += p[d];
    }
    for (int i = 0; i < DEG; ++i) c[i] = p[i];
}

constexpr Tables make_tables() {
    Tables t{};
    uint32_t r[313 + WINDOW] = {};
    r[0] = 1u;  // srand(0): glibc takes seed 0 as 1
    for (int i = 1; i < DEG; ++i) {
        // 16807 r mod (2^31 - 1) by Schrage's split, as glibc computes it (no 64-bit products)
        const int32_t word = (int32_t)r[i - 1];
        int32_t w = 16807 * (word % 127773) - 2836 * (word / 127773);
        if (w < 0) w += 2147483647;
        r[i] = (uint32_t)w;
    }
    for (int i = DEG; i < 34; ++i) r[i] = r[i - DEG];
    for (int i = 34; i < 313 + WINDOW; ++i) r[i] = r[i - 31] + r[i - 3];
    for (int i = 0; i < WINDOW; ++i) t.start[i] = r[313 + i];
    uint32_t c[DEG] = {};
    c[0] = 1u;  // x^31 = x^28 + 1
    c[28] = 1u;
    for (int k = 0; k < 5; ++k) square(c);
    for (int k = 0; k < MAX_JUMPS; ++k) {
        for (int i = 0; i < DEG; ++i) t.jump[k][i] = c[i];
        if (k + 1 < MAX_JUMPS) square(c);
    }
    return t;
}

__constant__ Tables g_tables = make_tables();

__host__ __device__ constexpr uint32_t binomial(int m, int k) {
    uint64_t b = 1;
    for (int i = 0; i < k; ++i) b = b * (uint64_t)(m - i) / (uint64_t)(i + 1);
    return (uint32_t)b;
}

// s[from .. to) from the 31 M values before `from`, 3 M at a time.
template <int M>
__device__ __forceinline__ void grow(uint32_t *s, int from, int to, int lane) {
    for (int i = from + lane; i - lane < to; i += 3 * M) {
        if (lane < 3 * M && i < to) {
            uint32_t v = 0u;
#pragma unroll
            for (int k = 0; k <= M; ++k) v += binomial(M, k) * s[i - DEG * M + 28 * k];
            s[i] = v;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(32 * WARPS) rand_init_kernel(int64_t total, float *__restrict__ V) {
    __shared__ uint32_t stretch[WARPS][STRETCH + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b = (int64_t)blockIdx.x * WARPS + warp;
    const int64_t beg = b * WARP_CALLS;
    if (beg >= total) return;
    uint32_t *s = stretch[warp];
    for (int i = lane; i < WINDOW; i += 32) s[i] = g_tables.start[i];
    __syncwarp();
    for (int k = 0; k < MAX_JUMPS && (b >> k); ++k) {
        if (!((b >> k) & 1)) continue;  // (warp-uniform)
        uint32_t v = 0u;
        if (lane < DEG) {
#pragma unroll
            for (int j = 0; j < DEG; ++j) v += g_tables.jump[k][j] * s[lane + j];
        }
        __syncwarp();
        if (lane < DEG) s[lane] = v;
        __syncwarp();
        grow<1>(s, DEG, WINDOW, lane);
    }
    const int64_t left = total - beg;
    const int end = DEG + (int)(left < WARP_CALLS ? left : WARP_CALLS);
    grow<1>(s, WINDOW, 62, lane);
    grow<2>(s, 62, 124, lane);
    grow<4>(s, 124, 248, lane);
    grow<8>(s, 248, end, lane);
    for (int i = DEG + lane; i < end; i += 32) {
        const float q = (float)(int32_t)(s[i] >> 1) / 2147483648.0f;  // (float)RAND_MAX
        V[beg + i - DEG] = (float)(0.2 * (double)q);
    }
}

}  // namespace

cudaError_t init_factors_device(int64_t m, int64_t n, int f, float *U, float *V,
                                cudaStream_t st) {
    const int64_t total = n * (int64_t)f;
    cudaError_t e = cudaMemsetAsync(U, 0, sizeof(float) * (size_t)(m * f), st);
    if (e != cudaSuccess || total <= 0) return e;
    const int64_t per_cta = (int64_t)WARPS * WARP_CALLS;
    rand_init_kernel<<<(unsigned)((total + per_cta - 1) / per_cta), 32 * WARPS, 0, st>>>(total, V);
    return cudaGetLastError();
}

}  // namespace als
