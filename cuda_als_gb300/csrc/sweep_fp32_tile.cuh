// sweep_fp32_tile.cuh — the FP32 half-sweep kernels for f <= 175, the matrix in registers
// (tilesolve.cuh): one CTA a row, heavy rows in parts.  Instantiated per panel pitch by
// sweep_fp32_p*.cu; sweep_fp32.cu picks between these and the wide kernels.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <algorithm>

#include "internal.h"
#include "solvers.cuh"
#include "tilesolve.cuh"

namespace als {

enum { TILE_LDLT = 0, TILE_LU = 1 };

// Threads: one a tile, or enough for the Gram's patches.
template <int P>
inline int tile_threads(int f, int mode) {
    const int nb = tile::nb_of(f);
    return std::max(tile::up32(mode == TILE_LU ? nb * nb : 0), tile::gram_threads(f, tile::patched<P>()));
}
template <int P>
inline size_t tile_smem(int f, int mode) {
    return sizeof(float) * tile::shared_floats<P>(tile::nb_of(f), mode == TILE_LU);
}
template <int P>
inline size_t part_smem() {
    return sizeof(float) * (tile::RING * tile::KCH * P + tile::RING * tile::KCH);
}
inline size_t tile_part_floats(int f) {
    const int nb = tile::nb_of(f);
    return 64 * (size_t)tile::tiles_of(nb) + 16 * (size_t)nb;
}

// From the finished Gram tiles and the rhs_threads' two columns of the right-hand side: regularise,
// solve, write x (or x = 0 and a flag).
template <int MODE, int P>
__device__ __forceinline__ void tile_solve(const SweepArgs &a, int nb, int row, int nu,
                                           tile::Acc &acc, const tile::Tile &t, float2 b,
                                           float *smem) {
    const int f = a.f, tid = threadIdx.x;
    const int rt = tile::rhs_thread(tile::patched<P>(), nb);
    const bool rhs = tile::rhs_columns(rt, f);
    float *xo = a.X + (int64_t)row * f;
    tile::add_diagonal(acc, t, f, (float)nu * a.lambda);  // items_cnt * lambda (als_model.cu:157-159)
    const tile::Shared s = tile::carve<P>(smem, nb, MODE == TILE_LU);
    if (tid == 0) *s.bad = 0;
    if (rhs) *reinterpret_cast<float2 *>(s.vb + 2 * rt) = b;
    for (int i = f + (f & 1) + tid; i < 8 * nb; i += blockDim.x) s.vb[i] = 0.f;
    if (MODE == TILE_LU) tile::mirror(acc, t, nb, s);
    __syncthreads();
    bool ok = tile::factor<MODE == TILE_LU, P>(acc, t, f, nb, s);
    if (ok) tile::backward<MODE == TILE_LU>(s.vb, s.vx, f, nb, s);
    int bad = 0;
    for (int i = tid; ok && i < f; i += blockDim.x) bad |= isfinite(s.vx[i]) ? 0 : 1;
    if (__syncthreads_or(bad)) ok = false;
    for (int i = tid; i < f; i += blockDim.x) xo[i] = ok ? s.vx[i] : 0.f;
    if (!ok && tid == 0 && a.flags) atomicAdd(&a.flags[0], 1);
}

template <int MODE, int P>
__global__ void __launch_bounds__(512) sweep_tile_kernel(const SweepArgs a, const int nb) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x;
    const int slot = a.row_begin + blockIdx.x;
    const int row = a.order ? a.order[slot] : slot;
    const int beg = a.ptr[row], end = a.ptr[row + 1], nu = end - beg;
    if (nu == 0) {  // no ratings: defined as x = 0 (the reference's LU would divide by zero)
        for (int i = tid; i < a.f; i += blockDim.x) a.X[(int64_t)row * a.f + i] = 0.f;
        return;
    }
    const tile::Tile t = tile::tile_of<P>(tid, nb, MODE == TILE_LU);
    tile::Acc acc;
    tile::clear(acc);
    float2 bsum = make_float2(0.f, 0.f), bcomp = bsum;
    tile::accumulate<P>(a.idx, a.val, a.Y, a.f, nb, beg, end, t, t.on && t.bi >= t.bj, acc, bsum, bcomp,
                        smem, smem + tile::big_floats<P>(nb, true));
    tile_solve<MODE, P>(a, nb, row, nu, acc, t, make_float2(bsum.x - bcomp.x, bsum.y - bcomp.y), smem);
}

// Heavy rows: part p accumulates ratings [beg[p], end[p]) of its row and stores its tiles (16
// float4 a tile, the same one of every thread side by side) and its compensated right-hand side.
template <int P>
__global__ void __launch_bounds__(512)
    gram_part_kernel(const SweepArgs a, const int nb, const int32_t *__restrict__ part_beg,
                     const int32_t *__restrict__ part_end, float *__restrict__ part) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, T = tile::tiles_of(nb), p = blockIdx.x;
    const tile::Tile t = tile::tile_of<P>(tid, nb, false);
    tile::Acc acc;
    tile::clear(acc);
    float2 bsum = make_float2(0.f, 0.f), bcomp = bsum;
    tile::accumulate<P>(a.idx, a.val, a.Y, a.f, nb, part_beg[p], part_end[p], t, t.on, acc, bsum,
                        bcomp, smem, smem + tile::RING * tile::KCH * P);
    float *out = part + (int64_t)p * (64 * (int64_t)T + 16 * nb);
    if (t.on) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int h = 0; h < 4; ++h)
                reinterpret_cast<ulonglong2 *>(out)[(4 * q + h) * T + tid] =
                    make_ulonglong2(acc[q][2 * h], acc[q][2 * h + 1]);
    }
    const int rt = tile::rhs_thread(tile::patched<P>(), nb);
    if (tile::rhs_columns(rt, a.f)) {
        *reinterpret_cast<float2 *>(out + 64 * (int64_t)T + 2 * rt) = bsum;
        *reinterpret_cast<float2 *>(out + 64 * (int64_t)T + 8 * nb + 2 * rt) = bcomp;
    }
}

// Heavy row at order position h: its parts first[h]..first[h+1] added in order (the tiles
// plainly, the right-hand sides with compensation), then the common regularise / solve / write.
template <int MODE, int P>
__global__ void __launch_bounds__(512)
    combine_solve_kernel(const SweepArgs a, const int nb, const int32_t *__restrict__ first,
                         const float *__restrict__ part) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, T = tile::tiles_of(nb), h = blockIdx.x;
    const int row = a.order ? a.order[h] : h;
    const int nu = a.ptr[row + 1] - a.ptr[row];
    const tile::Tile t = tile::tile_of<P>(tid, nb, MODE == TILE_LU);
    float sum[4][16];  // the pairs of acc
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 16; ++c) sum[q][c] = 0.f;
    float2 bsum = make_float2(0.f, 0.f), bcomp = bsum, blost = bsum;
    const int64_t stride = 64 * (int64_t)T + 16 * nb;
    const int rt = tile::rhs_thread(tile::patched<P>(), nb);
    for (int32_t p = first[h]; p < first[h + 1]; ++p) {
        const float *in = part + (int64_t)p * stride;
        if (tid < T) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const float4 v = reinterpret_cast<const float4 *>(in)[(4 * q + g) * T + tid];
                    sum[q][4 * g] += v.x;
                    sum[q][4 * g + 1] += v.y;
                    sum[q][4 * g + 2] += v.z;
                    sum[q][4 * g + 3] += v.w;
                }
        }
        if (tile::rhs_columns(rt, a.f)) {
            const float2 b = *reinterpret_cast<const float2 *>(in + 64 * (int64_t)T + 2 * rt);
            const float2 c = *reinterpret_cast<const float2 *>(in + 64 * (int64_t)T + 8 * nb + 2 * rt);
            const float y0 = b.x - bcomp.x, y1 = b.y - bcomp.y;
            const float t0 = bsum.x + y0, t1 = bsum.y + y1;
            bcomp = make_float2((t0 - bsum.x) - y0, (t1 - bsum.y) - y1);
            bsum = make_float2(t0, t1);
            blost.x += c.x;
            blost.y += c.y;
        }
    }
    tile::Acc acc;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[q][c] = tile::pack2(sum[q][2 * c], sum[q][2 * c + 1]);
    tile_solve<MODE, P>(a, nb, row, nu, acc, t,
                        make_float2((bsum.x - bcomp.x) - blost.x, (bsum.y - bcomp.y) - blost.y), smem);
}

template <int MODE, int P>
cudaError_t launch_tiles(const SweepArgs &a, const Fp32Split *sp, cudaStream_t st, int *launches) {
    const int nb = tile::nb_of(a.f), nt = tile_threads<P>(a.f, MODE);
    const int ntp = tile::gram_threads(a.f, tile::patched<P>());
    const size_t smem = tile_smem<P>(a.f, MODE);
    if (smem > 48 * 1024) {  // (a part's ring stays below)
        cudaError_t e = cudaFuncSetAttribute(sweep_tile_kernel<MODE, P>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(combine_solve_kernel<MODE, P>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    SweepArgs b = a;
    // the heavy rows are the first order positions: split when the slice starts there
    if (sp && sp->nheavy > 0 && a.row_begin == 0 && a.order) {
        const int32_t nh = sp->nheavy < a.row_end ? sp->nheavy : a.row_end;
        gram_part_kernel<P><<<(unsigned)sp->first_host[nh], ntp, part_smem<P>(), st>>>(
            a, nb, sp->part_beg, sp->part_end, sp->part);
        combine_solve_kernel<MODE, P><<<(unsigned)nh, nt, smem, st>>>(a, nb, sp->first, sp->part);
        if (launches) *launches += 2;
        b.row_begin = nh;
    }
    const int n = b.row_end - b.row_begin;
    if (n > 0) {
        // Up to eight rows an SM are a matter of latency: another warp shares the copies and, at
        // f <= 16, takes the right-hand side over.  With more rows it would take CTAs' places.
        // 1,000 x 500, f = 10, ten epochs: 0.57 -> 0.48 ms a training call; f = 24, 1,000 rows 53 ->
        // 47 us.
        const int more = tile::patched<P>() && n <= 8 * 152 ? 32 : 0;
        sweep_tile_kernel<MODE, P><<<(unsigned)n, nt + more, smem, st>>>(b, nb);
        if (launches) ++*launches;
    }
    return cudaGetLastError();
}

template <int P>
cudaError_t launch_tiles_of(const SweepArgs &a, const Fp32Split *sp, cudaStream_t st, int *launches) {
    return a.solve == ALS_SOLVE_LU ? launch_tiles<TILE_LU, P>(a, sp, st, launches)
                                   : launch_tiles<TILE_LDLT, P>(a, sp, st, launches);
}

#define ALS_FP32_TILES(P)                                                                        \
    cudaError_t launch_tiles_##P(const SweepArgs &a, const Fp32Split *sp, cudaStream_t st,       \
                                 int *launches)
ALS_FP32_TILES(32);
ALS_FP32_TILES(64);
ALS_FP32_TILES(128);
ALS_FP32_TILES(192);

}  // namespace als
