// The register-tile solvers' arithmetic against CUDA's division and against the column-at-a-time
// solvers: bit for bit while pivots are in quotient's range, else by their errors against FP64.  argv[1]: "reciprocal", "quotients" or "solve"; prints "<what> <compared>
// <different>" lines.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "sweep_fp32_tile.cuh"

using namespace als;

#define CHECK(x)                                                                   \
    do {                                                                           \
        const cudaError_t e_ = (x);                                                \
        if (e_ != cudaSuccess) {                                                   \
            std::fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_));          \
            return 1;                                                              \
        }                                                                          \
    } while (0)

__device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// Every significand at exponent e, both signs.
__global__ void reciprocals(int e, unsigned long long *bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const float x = __uint_as_float((i >> 23) << 31 | (uint32_t)(127 + e) << 23 | (i & 0x7fffffu));
    if (!same(tile::reciprocal(x), 1.0f / x)) atomicAdd(bad, 1ull);
}

__device__ uint32_t mix(uint32_t x) {  // (a 32-bit finaliser: Prospecting, C. Wellons, 2018)
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return x ^ (x >> 16);
}

// Quotients in quotient's range: exponents of any size, within `span` of 1, or the range's edges.
__global__ void divisions(uint32_t seed, int span, unsigned long long *count) {
    uint32_t s = mix(seed ^ mix(blockIdx.x * blockDim.x + threadIdx.x + 1u));
    auto value = [&]() -> float {
        s = mix(s + 0x9e3779b9u);
        uint32_t x = s & 0x7fffffffu;
        if (span > 0) x = (127u - span + mix(s) % (2u * span + 1u)) << 23 | (x & 0x7fffffu);
        if (span < 0) {  // 0, 2^-102, 2^-100, 1 and 2^100, and their neighbours
            const uint32_t edge[] = {0u, 25u << 23, 27u << 23, 127u << 23, 227u << 23};
            x = edge[mix(s) % 5u];
            if (x) x += mix(s ^ 3u) % 3u - 1u;
        }
        return __uint_as_float(x | (mix(s ^ 5u) & 0x80000000u));
    };
    unsigned long long n = 0, bad = 0;
    for (int k = 0; k < 128; ++k) {
        const float a = value(), d = fabsf(value()), q = a / d;
        if (!(d >= 0x1p-100f && d <= 0x1p100f)) continue;
        if (!(a == 0.f || (fabsf(a) >= 0x1p-102f && fabsf(q) >= 0x1p-126f && fabsf(q) < 0x1p127f))) continue;
        const float got = tile::quotient(a, d, 1.0f / d);
        ++n;
        bad += a == 0.f ? got != 0.f : !same(got, q);
    }
    atomicAdd(count, n);
    if (bad) atomicAdd(count + 1, bad);
}

template <int MODE, int P>
__global__ void __launch_bounds__(512) by_tiles(const float *A, const float *b, int f, int nb, float *x, int *ok) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x;
    const tile::Tile t = tile::tile_of<P>(tid, nb, MODE == TILE_LU);
    const tile::Shared s = tile::carve<P>(smem, nb, MODE == TILE_LU);
    float m[8][8];
    for (int r = 0; r < 8; ++r)
        for (int c = 0; c < 8; ++c) {
            const int i = 8 * t.bi + r, j = 8 * t.bj + c;
            m[r][c] = t.on && i < f && j < f ? A[i * f + j] : 0.f;
        }
    tile::Acc acc;
    tile::repack(m, acc);
    for (int i = tid; i < 8 * nb; i += blockDim.x) s.vb[i] = i < f ? b[i] : 0.f;
    if (tid == 0) *s.bad = 0;
    __syncthreads();
    const bool good = tile::factor<MODE == TILE_LU, P>(acc, t, f, nb, s);
    if (good) tile::backward<MODE == TILE_LU>(s.vb, s.vx, f, nb, s);
    for (int i = tid; i < f; i += blockDim.x) x[i] = good ? s.vx[i] : 0.f;
    if (tid == 0) *ok = good;
}

template <int MODE>
__global__ void by_columns(const float *A, const float *b, int f, float *x, int *ok) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, nt = blockDim.x, gs = f + 1;
    float *G = smem, *v = smem + f * gs;
    for (int e = tid; e < f * f; e += nt) G[e / f * gs + e % f] = A[e];
    for (int i = tid; i < f; i += nt) v[i] = b[i];
    __syncthreads();
    bool good;
    if (MODE == TILE_LU) {
        good = lu_nopivot_solve<CtaSync>(G, gs, f, v, tid, nt);
    } else {
        good = ldlt_factor<CtaSync>(G, gs, f, tid, nt);
        if (good) ldlt_solve<CtaSync>(G, gs, f, v, tid);
    }
    __syncthreads();
    for (int i = tid; i < f; i += nt) x[i] = good ? v[i] : 0.f;
    if (tid == 0) *ok = good;
}

// ||x - X|| / ||X|| with A X = b by Cholesky in FP64; infinite if x is not finite.
static double error_of(const float *A, const float *b, int f, const float *x) {
    std::vector<double> L((size_t)f * f), X(f);
    for (int i = 0; i < f; ++i)
        for (int j = 0; j <= i; ++j) {
            double s = A[i * f + j];
            for (int k = 0; k < j; ++k) s -= L[i * f + k] * L[j * f + k];
            L[i * f + j] = i == j ? std::sqrt(s) : s / L[j * f + j];
        }
    for (int i = 0; i < f; ++i) {
        double s = b[i];
        for (int k = 0; k < i; ++k) s -= L[i * f + k] * X[k];
        X[i] = s / L[i * f + i];
    }
    for (int i = f - 1; i >= 0; --i) {
        double s = X[i];
        for (int k = i + 1; k < f; ++k) s -= L[k * f + i] * X[k];
        X[i] = s / L[i * f + i];
    }
    double d = 0.0, n = 0.0;
    for (int i = 0; i < f; ++i) {
        d += (x[i] - X[i]) * (x[i] - X[i]);
        n += X[i] * X[i];
    }
    return std::isfinite(d) ? std::sqrt(d / n) : INFINITY;
}

template <int MODE, int P>
cudaError_t solve_both(const float *A, const float *b, int f, float *x, int *ok) {
    const int nb = tile::nb_of(f);
    const size_t st = tile_smem<P>(f, MODE), sc = sizeof(float) * (size_t)f * (f + 2);
    cudaError_t e = cudaFuncSetAttribute(by_tiles<MODE, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)st);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(by_columns<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sc);
    if (e != cudaSuccess) return e;
    by_tiles<MODE, P><<<1, tile_threads<P>(f, MODE), st>>>(A, b, f, nb, x, ok);
    by_columns<MODE><<<1, 256, sc>>>(A, b, f, x + f, ok + 1);
    return cudaGetLastError();
}
template <int MODE>
cudaError_t solve_both(const float *A, const float *b, int f, float *x, int *ok) {
    switch (tile::pitch_of(f)) {
    case 32: return solve_both<MODE, 32>(A, b, f, x, ok);
    case 64: return solve_both<MODE, 64>(A, b, f, x, ok);
    case 128: return solve_both<MODE, 128>(A, b, f, x, ok);
    default: return solve_both<MODE, 192>(A, b, f, x, ok);
    }
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    unsigned long long *bad, n = 0;
    CHECK(cudaMallocManaged(&bad, 2 * sizeof(*bad)));
    if (what == "reciprocal") {
        for (int e : {-100, -99, -1, 0, 1, 57, 99}) {
            *bad = 0;
            reciprocals<<<1 << 16, 256>>>(e, bad);
            CHECK(cudaDeviceSynchronize());
            std::printf("2^%d %u %llu\n", e, 1u << 24, *bad);
        }
        return 0;
    }
    if (what == "quotients") {
        for (int span : {0, 1, 20, 60, 99, 102, 126, -1}) {
            bad[0] = bad[1] = 0;
            divisions<<<1 << 12, 256>>>(17u + (uint32_t)span, span, bad);
            CHECK(cudaDeviceSynchronize());
            std::printf("span%d %llu %llu\n", span, bad[0], bad[1]);
        }
        return 0;
    }
    if (what != "solve") return 2;
    std::mt19937 rng(7);
    std::normal_distribution<double> normal;
    float *A, *b, *x;
    int *ok;
    CHECK(cudaMallocManaged(&A, sizeof(float) * 176 * 176));
    CHECK(cudaMallocManaged(&b, sizeof(float) * 176));
    CHECK(cudaMallocManaged(&x, sizeof(float) * 2 * 176));
    CHECK(cudaMallocManaged(&ok, sizeof(int) * 2));
    // scale: of the whole matrix, 2^scale; spread: row and column i also by 2^(-spread .. spread)
    const int scales[][2] = {{0, 0}, {-52, 0}, {-62, 0}, {-96, 0}, {-110, 0}, {-124, 0}, {-140, 0}, {62, 0},
                             {96, 0}, {110, 0}, {123, 0}, {0, 12}, {0, 30}, {0, 45}, {0, 60}};
    for (int lu = 0; lu < 2; ++lu) {
        for (const auto &sc : scales) {
            unsigned long long diff = 0;
            n = 0;
            for (int f : {1, 2, 5, 8, 9, 20, 32, 33, 63, 64, 65, 100, 128, 129, 150, 175}) {
                const int k = f + f / 2 + 3;
                std::vector<double> Y((size_t)k * f);
                for (auto &v : Y) v = 0.3 * normal(rng);
                std::vector<int> sh(f);
                for (auto &v : sh) v = sc[1] ? (int)(rng() % (2 * sc[1] + 1)) - sc[1] : 0;
                for (int i = 0; i < f; ++i) {
                    for (int j = 0; j <= i; ++j) {
                        double s = i == j ? 0.05 * k : 0.0;
                        for (int q = 0; q < k; ++q) s += Y[(size_t)q * f + i] * Y[(size_t)q * f + j];
                        A[i * f + j] = A[j * f + i] = (float)std::ldexp(s, sc[0] + sh[i] + sh[j]);
                    }
                    b[i] = (float)std::ldexp(normal(rng), sc[0] / 2 + sh[i]);
                }
                CHECK(lu ? solve_both<TILE_LU>(A, b, f, x, ok) : solve_both<TILE_LDLT>(A, b, f, x, ok));
                CHECK(cudaDeviceSynchronize());
                diff += ok[0] != ok[1];
                const bool in_range = std::abs(sc[0]) <= 96 && sc[1] <= 45;  // (pivots within 2^4 of the scales)
                if (!in_range) {  // no further from FP64 than half as much again
                    ++n;
                    if (ok[0] && ok[1]) diff += error_of(A, b, f, x) > 1.5 * error_of(A, b, f, x + f) + 1e-7;
                    continue;
                }
                for (int i = 0; i < f; ++i, ++n)
                    diff += std::memcmp(x + i, x + f + i, sizeof(float)) != 0 && !(x[i] != x[i] && x[f + i] != x[f + i]);
            }
            std::printf("%s_%d_%d %llu %llu\n", lu ? "lu" : "ldlt", sc[0], sc[1], n, diff);
        }
    }
    return 0;
}
