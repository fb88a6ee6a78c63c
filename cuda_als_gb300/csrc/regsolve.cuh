// regsolve.cuh — register-resident per-row solvers for the tensor-core epilogue.
//
// After tcgen05.ld, thread i of a 128-thread solver warpgroup holds row i of the (padded) Gram
// A in registers (a[0..FP)), and b_i.  Rows f <= i < FP are padded with the identity, so every
// solver runs at the compile-time size FP (a multiple of 16) and leaves x_i = 0 there.  Threads
// with i >= FP (FP < 128) hold zero rows: they join every barrier and shuffle but never index
// shared memory with i.
//
//   cg_reg        warm-started CG of cumf_als_cg/cg.cu:37-232 (same recurrences, same exit rule
//                 r'r < tol); the matvec reads p from shared memory as float4 broadcasts.
//   cg_quad       the same CG with four rows shared by a lane quad (half of them in shared
//                 memory): a quarter of the p reads, for rows too long to keep in registers.
//   chol_fac      Cholesky A = L L^T of the Gram copied to a packed lower triangle in shared
//                 memory, left-looking in blocks of 8 columns, with the forward solve beside it:
//                 the dot products are spread over the threads as (row, column half) items,
//                 every lane of one warp factors each 8 x 8 diagonal block in registers and eight
//                 of them invert it, two barriers per block.
//   chol_forward, chol_backward  L y = b and L^T x = y by the group, one barrier per 16 rows.
// Sums over threads are combined in a fixed order (deterministic).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace als {

struct GroupSync {
    int id;
    __device__ void sync() const { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
};

// Fixed-order sum over the 128 threads; `red` is a 4 x 4 float ring in shared memory, `slot`
// rotates so that consecutive calls never overwrite values still being read.
__device__ __forceinline__ float gsum128(float v, float *red, int &slot, const GroupSync &gs) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    float *r = red + 4 * (slot & 3);
    ++slot;
    if ((threadIdx.x & 31) == 0) r[((threadIdx.x >> 5) & 3)] = v;
    gs.sync();
    return (r[0] + r[1]) + (r[2] + r[3]);
}

// Two fixed-order sums over the 128 threads in one pass (one barrier); `red` as for gsum128 (the
// two values of a warp share a float2 of the same ring slot: 4 x 8 floats).
__device__ __forceinline__ float2 gsum128x2(float u, float v, float *red, int &slot,
                                            const GroupSync &gs) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    float2 *r = reinterpret_cast<float2 *>(red) + 4 * (slot & 3);
    ++slot;
    if ((threadIdx.x & 31) == 0) r[((threadIdx.x >> 5) & 3)] = make_float2(u, v);
    gs.sync();
    const float2 a = r[0], b = r[1], c = r[2], d = r[3];
    return make_float2((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y));
}

__device__ __forceinline__ float gmax128(float v, float *red, int &slot, const GroupSync &gs) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    float *r = red + 4 * (slot & 3);
    ++slot;
    if ((threadIdx.x & 31) == 0) r[((threadIdx.x >> 5) & 3)] = v;
    gs.sync();
    return fmaxf(fmaxf(r[0], r[1]), fmaxf(r[2], r[3]));
}

// warp index inside the warpgroup that owns TMEM lanes [32w, 32w+32): tcgen05 lane quarters
// follow warp_id % 4, so thread i of the row space is (warp % 4) * 32 + lane.
template <int FP>
__device__ __forceinline__ float dot_row(const float (&a)[FP], const float *sv) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
    for (int j = 0; j < FP; j += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(sv + j);
        s0 = fmaf(a[j], v.x, s0);
        s1 = fmaf(a[j + 1], v.y, s1);
        s2 = fmaf(a[j + 2], v.z, s2);
        s3 = fmaf(a[j + 3], v.w, s3);
    }
    return (s0 + s1) + (s2 + s3);
}

// CG with one reduction per iteration (Chronopoulos and Gear, 1989): with w = A r, the two dot
// products gamma = r'r and delta = r'w are summed together, and p'Ap = delta - beta gamma / alpha
// follows from the recurrences.  In exact arithmetic the iterates are those of the reference's
// CG (cumf_als_cg/cg.cu:37-232, warm start, at most `iters` updates, exit when r'r < tol after an
// update, stop before an update whose p'Ap is not positive); a product of A follows every update
// but the last, so without an early exit it performs the same iters + 1 products, with one
// barrier and one two-value reduction per iteration instead of three barriers and two
// reductions.  `mul(v)` returns (A v)_i after publishing v_i to the group (it synchronises).
template <class Mul>
__device__ __forceinline__ float cg_single_reduction(Mul mul, float bi, float xi, float *red,
                                                     int iters, float tol, const GroupSync &gs) {
    int slot = 0;
    float r = bi - mul(xi);
    gs.sync();  // every thread has read x out of the shared vector before r overwrites it
    float w = mul(r);
    float2 gd = gsum128x2(r * r, r * w, red, slot, gs);
    float gamma = gd.x, pap = gd.y;
    float p = r, s = w, alpha = 0.f;
    for (int it = 0; it < iters; ++it) {
        if (!(pap > 0.f)) break;
        alpha = gamma / pap;
        xi = fmaf(alpha, p, xi);
        r = fmaf(-alpha, s, r);
        if (it + 1 == iters) break;  // no further update: the product would be unused
        w = mul(r);
        gd = gsum128x2(r * r, r * w, red, slot, gs);
        if (gd.x < tol) break;
        const float beta = gd.x / gamma;
        pap = gd.y - beta * gd.x / alpha;  // p_new' A p_new
        gamma = gd.x;
        p = fmaf(beta, p, r);
        s = fmaf(beta, s, w);
    }
    return xi;
}

template <int FP>
__device__ float cg_reg(const float (&a)[FP], float bi, float xi, int i, float *sv, float *red,
                        int iters, float tol, const GroupSync &gs) {
    const bool live = i < FP;  // threads past the padded size hold zero rows and write nothing
    auto mul = [&](float v) -> float {
        if (live) sv[i] = v;  // every thread finished reading sv at the previous reduction
        gs.sync();
        return dot_row<FP>(a, sv);
    };
    return cg_single_reduction(mul, bi, xi, red, iters, tol, gs);
}

// CG as cg_reg with the rows quad-blocked (FP = 64, 112, 128).  The four lanes 4a..4a+3 of a warp share
// rows 4a..4a+3: lane 4a+c holds columns 16k+4c..16k+4c+3 (k < NK = FP/16) of all four, rows 4a
// and 4a+1 in registers (ar[0], ar[1]), rows 4a+2 and 4a+3 in shared memory (slots 2k and 2k+1
// of `sa`, the thread's own float4 in each).  A product reads FP/4 floats of p a thread, one
// float4 per chunk shared by the four rows, where a whole row a thread needs all FP of them; the
// quad's partial sums are then reduced and scattered so that lane 4a+c ends with row 4a+c.
constexpr int CGQ_SLOT = 130;  // float4 a slot: 128 threads + 2 (staggers the slots' banks)

__device__ __forceinline__ float4 shfl_xor4(float4 v, int m) {
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m),
                       __shfl_xor_sync(0xffffffffu, v.z, m), __shfl_xor_sync(0xffffffffu, v.w, m));
}

template <int NK>
__device__ __forceinline__ float dot_quad(const float4 (&ar)[2][NK], const float4 *sa,
                                          const float *sv, int t) {
    const int c = t & 3;
    const float4 *pv = reinterpret_cast<const float4 *>(sv) + c;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
        const float4 v = pv[4 * k];
        const float4 s2 = sa[(2 * k) * CGQ_SLOT + t];
        const float4 s3 = sa[(2 * k + 1) * CGQ_SLOT + t];
        a0 = fmaf(ar[0][k].x, v.x, fmaf(ar[0][k].y, v.y, fmaf(ar[0][k].z, v.z, fmaf(ar[0][k].w, v.w, a0))));
        a1 = fmaf(ar[1][k].x, v.x, fmaf(ar[1][k].y, v.y, fmaf(ar[1][k].z, v.z, fmaf(ar[1][k].w, v.w, a1))));
        a2 = fmaf(s2.x, v.x, fmaf(s2.y, v.y, fmaf(s2.z, v.z, fmaf(s2.w, v.w, a2))));
        a3 = fmaf(s3.x, v.x, fmaf(s3.y, v.y, fmaf(s3.z, v.z, fmaf(s3.w, v.w, a3))));
    }
    // reduce-scatter over the quad: lanes c, c^2 combine rows {0,1} (c < 2) or {2,3}, then
    // lanes c, c^1 combine row c
    const bool hi = (c & 2) != 0;
    float k0 = hi ? a2 : a0, k1 = hi ? a3 : a1;
    const float s0 = hi ? a0 : a2, s1 = hi ? a1 : a3;
    k0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    k1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    const bool odd = (c & 1) != 0;
    return (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 1);
}

// The quad-blocked rows hold the Gram without its diagonal term: thread i adds dreg * v_i (lambda
// n_u, or 1 on a padded row, whose Gram row is zero) to each product.
template <int NK>
__device__ float cg_quad(const float4 (&ar)[2][NK], const float4 *sa, float bi, float xi, int i,
                         float *sv, float *red, int iters, float tol, const GroupSync &gs,
                         float dreg) {
    constexpr int FP = 16 * NK;
    const bool live = i < FP;
    auto mul = [&](float v) -> float {
        if (live) sv[i] = v;
        gs.sync();
        return fmaf(dreg, v, dot_quad<NK>(ar, sa, sv, i));
    };
    return cg_single_reduction(mul, bi, xi, red, iters, tol, gs);
}

// Packed lower triangle of an FP x FP factor in shared memory.  Row i (block K = i / 8) keeps
// columns 0 .. 8(K+1)-1, so every 8 x 8 block a row touches is whole; rows are laid out one
// after the other with 4 floats of skew each, which keeps the float4 loads of 8 consecutive
// rows on distinct banks.  Offsets are multiples of 4 floats (16-byte aligned float4 access).
__device__ __forceinline__ int tri_off(int i) {
    const int K = i >> 3;
    return 8 * (K + 1) * (4 * K + (i & 7)) + 4 * i;
}
template <int FP>
struct TriLayout {
    static constexpr int floats = 32 * (FP / 8) * (FP / 8 + 1) + 4 * FP;
};

// Cholesky A = L L^T of the leading n x n matrix (n a multiple of 16) held in Ls (packed, tri_off
// rows; entry (i, j) for j <= i must be set, the rest of each row's blocks is scratch), and the
// forward solve L y = b beside it: `bv` holds b on entry (n floats, scratch afterwards), `yv`
// receives y.  On exit entry (i, j) left of the diagonal blocks holds L[i][j],
// Dv[K * 64 + r * 8 + c] = (L_KK^-1)[r][c] for r >= c (the inverse of each 8 x 8 diagonal block) and
// invd[j] = 1 / L[j][j].  Called by the 128 threads of a group (et = 0..127); warp `lead` / 32 works
// on the diagonal blocks.
//
// Left-looking in blocks of 8 columns, two barriers per block:
//  (a) the block's entries lose L[r][0:k0] . L[k0+4h+kk][0:k0], a (row, column half) item a thread,
//      the diagonal block's among the lead warp's, which goes on to (b) without waiting;
//  (b) the lead warp factors the 8 x 8 diagonal block in registers (rsqrt pivots), every lane alike,
//      so that eight of them have it at hand to invert it, a column each;
//  (c) every row below takes its block columns as s L_KK^-T; each thread also forms the block's
//      y = L_KK^-1 b and folds it into its own row's b.
// The groups' serial steps, (b) above all, set the time.  Work is dealt from the lead warp on, so
// that the groups' few busy warps sit on different schedulers.  Half-sweep over 480,189 rows and
// 98.6M ratings, ms at f = 64 / 100 / 128: 24.0 / 50.9 / 91.5 with separate solves and work dealt
// from warp 0 (and one buffer less at 128), then 18.0 / 36.1 / 51.8; with (b)'s factor no longer
// passed from one lane to the inverting ones through shared memory f = 64 15.8, and 100,000 rows of
// 9.0M ratings at f = 100 / 128 7.39 / 10.61 -> 6.69 / 9.50; with (b) beside the other warps' (a)
// f = 64 15.4, 100,000 rows 6.59 / 8.98.  Two rows an item in (a): 18.8 / 38.5 / 53.8; (a) for the
// next block by the warps that idle in (b): 19.1 / 38.2 / 50.5.
// Returns false (on the lead warp's lanes) if a pivot was not positive and finite.
__device__ __forceinline__ bool chol_fac(int et, int n, int lead, float *Ls, float *Dv, float *invd,
                                         float *bv, float *yv, const GroupSync &gs) {
    constexpr int B = 8;
    bool ok = true;
    const int ev = (et + 128 - lead) & 127;
#pragma unroll 1
    for (int K = 0; K < n / B; ++K) {
        const int k0 = K * B;
        if (k0 > 0) {
            const int nitems = 2 * (n - k0);
            for (int t = ev; t < nitems; t += ev < 32 ? nitems : 96) {
                const int r = k0 + (t >> 1), c0 = k0 + 4 * (t & 1);
                float *lr = Ls + tri_off(r);
                const float *l0 = Ls + tri_off(c0), *l1 = Ls + tri_off(c0 + 1);
                const float *l2 = Ls + tri_off(c0 + 2), *l3 = Ls + tri_off(c0 + 3);
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
                for (int q = 0; q < k0; q += 4) {
                    const float4 o = *reinterpret_cast<const float4 *>(lr + q);
                    const float4 a0 = *reinterpret_cast<const float4 *>(l0 + q);
                    const float4 a1 = *reinterpret_cast<const float4 *>(l1 + q);
                    const float4 a2 = *reinterpret_cast<const float4 *>(l2 + q);
                    const float4 a3 = *reinterpret_cast<const float4 *>(l3 + q);
                    s0 = fmaf(o.x, a0.x, s0); s1 = fmaf(o.x, a1.x, s1);
                    s2 = fmaf(o.x, a2.x, s2); s3 = fmaf(o.x, a3.x, s3);
                    s0 = fmaf(o.y, a0.y, s0); s1 = fmaf(o.y, a1.y, s1);
                    s2 = fmaf(o.y, a2.y, s2); s3 = fmaf(o.y, a3.y, s3);
                    s0 = fmaf(o.z, a0.z, s0); s1 = fmaf(o.z, a1.z, s1);
                    s2 = fmaf(o.z, a2.z, s2); s3 = fmaf(o.z, a3.z, s3);
                    s0 = fmaf(o.w, a0.w, s0); s1 = fmaf(o.w, a1.w, s1);
                    s2 = fmaf(o.w, a2.w, s2); s3 = fmaf(o.w, a3.w, s3);
                }
                float4 *d = reinterpret_cast<float4 *>(lr + c0);
                float4 v = *d;
                v.x -= s0; v.y -= s1; v.z -= s2; v.w -= s3;
                *d = v;
            }
            __syncwarp();
        }
        float *dv = Dv + K * B * B;
        if (ev < 32) {
            // (b) right-looking in registers, on every lane alike (a pivot that is not positive
            // leaves the rest undefined: the caller drops the row)
            float m[B][B], iv[B];
#pragma unroll
            for (int r = 0; r < B; ++r) {
                const float *lr = Ls + tri_off(k0 + r) + k0;
                const float4 x = *reinterpret_cast<const float4 *>(lr);
                m[r][0] = x.x; m[r][1] = x.y; m[r][2] = x.z; m[r][3] = x.w;
                if (r >= 4) {
                    const float4 y = *reinterpret_cast<const float4 *>(lr + 4);
                    m[r][4] = y.x; m[r][5] = y.y; m[r][6] = y.z; m[r][7] = y.w;
                }
            }
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const float dk2 = m[k][k];
                ok = ok && dk2 > 0.f && isfinite(dk2);
                iv[k] = rsqrtf(dk2);
#pragma unroll
                for (int r = k + 1; r < B; ++r) m[r][k] *= iv[k];
#pragma unroll
                for (int r = k + 1; r < B; ++r)
#pragma unroll
                    for (int j = k + 1; j <= r; ++j) m[r][j] = fmaf(-m[r][k], m[j][k], m[r][j]);
            }
            if (et == lead) {
                *reinterpret_cast<float4 *>(invd + k0) = make_float4(iv[0], iv[1], iv[2], iv[3]);
                *reinterpret_cast<float4 *>(invd + k0 + 4) = make_float4(iv[4], iv[5], iv[6], iv[7]);
            }
            // its inverse, lane c column c: D[c][c] = 1 / L_cc,
            // D[r][c] = -(sum_{c <= t < r} L[r][t] D[t][c]) / L[r][r]
            const int c = et & 31;
            float d[B];
#pragma unroll
            for (int r = 0; r < B; ++r) {
                float acc = 0.f;
#pragma unroll
                for (int t = 0; t < r; ++t) acc = fmaf(m[r][t], d[t], acc);  // (d[t < c] is zero)
                d[r] = r < c ? 0.f : r == c ? iv[r] : -acc * iv[r];
                if (c < B && r >= c) dv[r * B + c] = d[r];
            }
        }
        gs.sync();
        // (c) rows below the block; b's block by every thread, the first keeps it
        const int row = k0 + B + ev;
        if (row < n || ev == 0) {
            float rb[B], y[B], sb[B], o[B];
            const float4 b0 = *reinterpret_cast<const float4 *>(bv + k0);
            const float4 b1 = *reinterpret_cast<const float4 *>(bv + k0 + 4);
            rb[0] = b0.x; rb[1] = b0.y; rb[2] = b0.z; rb[3] = b0.w;
            rb[4] = b1.x; rb[5] = b1.y; rb[6] = b1.z; rb[7] = b1.w;
            float *lr = Ls + tri_off(row < n ? row : k0) + k0;
            const float4 x0 = *reinterpret_cast<const float4 *>(lr);
            const float4 x1 = *reinterpret_cast<const float4 *>(lr + 4);
            sb[0] = x0.x; sb[1] = x0.y; sb[2] = x0.z; sb[3] = x0.w;
            sb[4] = x1.x; sb[5] = x1.y; sb[6] = x1.z; sb[7] = x1.w;
#pragma unroll
            for (int kk = 0; kk < B; ++kk) {
                float acc = 0.f, accy = 0.f, dr[B];
                const float4 d0 = *reinterpret_cast<const float4 *>(dv + kk * B);
                const float4 d1 = *reinterpret_cast<const float4 *>(dv + kk * B + (kk >= 4 ? 4 : 0));
                dr[0] = d0.x; dr[1] = d0.y; dr[2] = d0.z; dr[3] = d0.w;
                dr[4] = d1.x; dr[5] = d1.y; dr[6] = d1.z; dr[7] = d1.w;
#pragma unroll
                for (int q = 0; q <= kk; ++q) {
                    acc = fmaf(sb[q], dr[q], acc);
                    accy = fmaf(dr[q], rb[q], accy);
                }
                o[kk] = acc;
                y[kk] = accy;
            }
            if (row < n) {
                *reinterpret_cast<float4 *>(lr) = make_float4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<float4 *>(lr + 4) = make_float4(o[4], o[5], o[6], o[7]);
                float t = bv[row];
#pragma unroll
                for (int q = 0; q < B; ++q) t = fmaf(-o[q], y[q], t);
                bv[row] = t;
            }
            if (ev == 0) {
                *reinterpret_cast<float4 *>(yv + k0) = make_float4(y[0], y[1], y[2], y[3]);
                *reinterpret_cast<float4 *>(yv + k0 + 4) = make_float4(y[4], y[5], y[6], y[7]);
            }
        }
        gs.sync();
    }
    return ok;
}

// The triangular solves by the whole group: thread t keeps the running value of row t.  Blocks of
// 16 rows, one barrier each: the warp that owns the rows solves the block's two 8-row halves with
// their inverses (lane l0 + c computes result c from shuffles of the rows' running values), folds
// the first half into its own later rows in between, and publishes the 16 results in `xb`; after
// the barrier every other row folds them into its own.  Each row sees the same FMA sequence as in
// a one-warp solve.  Blocks use the two 16-float halves of `xb` in turn, so a block's writer never
// overwrites values a thread has yet to read, from one solve to the next either.
__device__ __forceinline__ void fold8(const float *l, int stride, const float (&y)[8], float &t) {
#pragma unroll
    for (int q = 0; q < 8; ++q) t = fmaf(-l[q * stride], y[q], t);
}
__device__ __forceinline__ void read8(const float *p, float (&y)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    y[0] = a.x; y[1] = a.y; y[2] = a.z; y[3] = a.w;
    y[4] = b.x; y[5] = b.y; y[6] = b.z; y[7] = b.w;
}
// `acc` <- the row's y with L y = acc (et >= n: no row).
__device__ __forceinline__ void chol_forward(int et, int n, const float *Ls, const float *Dv, float *xb,
                                             float &acc, const GroupSync &gs) {
    const int lane = et & 31, w = et >> 5;
    const bool live = et < n;
    const float *own = Ls + tri_off(live ? et : 0);
#pragma unroll 1
    for (int b = 0; b < n / 16; ++b) {
        const int k0 = 16 * b;
        float *xk = xb + (b & 1) * 16;
        float y[8], l[8];
        if (w == (k0 >> 5)) {  // warp-uniform: the warp holding rows k0..k0+15
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int l0 = (k0 & 31) + 8 * h, c = lane - l0;
                float r[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) r[q] = __shfl_sync(0xffffffffu, acc, l0 + q);
                if (c >= 0 && c < 8) {
                    const float *dr = Dv + (2 * b + h) * 64 + c * 8;  // row c of the inverse, q <= c
                    float v = 0.f;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q <= c) v = fmaf(dr[q], r[q], v);
                    acc = v;
                    xk[8 * h + c] = v;
                }
                if (h == 0) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) y[q] = __shfl_sync(0xffffffffu, acc, l0 + q);
                    if (live && et >= k0 + 8) {
                        read8(own + k0, l);
                        fold8(l, 1, y, acc);
                    }
                }
            }
        }
        gs.sync();
        if (live && et >= k0 + 16) {
            if (w != (k0 >> 5)) {
                read8(xk, y);
                read8(own + k0, l);
                fold8(l, 1, y, acc);
            }
            read8(xk + 8, y);
            read8(own + k0 + 8, l);
            fold8(l, 1, y, acc);
        }
    }
}
// `acc` <- the row's x with L^T x = acc.
__device__ __forceinline__ void chol_backward(int et, int n, const float *Ls, const float *Dv, float *xb,
                                              float &acc, const GroupSync &gs) {
    const int lane = et & 31, w = et >> 5;
    auto fold = [&](int r0, const float (&x)[8]) {  // the results of rows r0..r0+7
#pragma unroll
        for (int q = 0; q < 8; ++q) acc = fmaf(-Ls[tri_off(r0 + q) + et], x[q], acc);
    };
#pragma unroll 1
    for (int b = n / 16 - 1; b >= 0; --b) {
        const int k0 = 16 * b;
        float *xk = xb + ((b + 1) & 1) * 16;
        float x[8];
        if (w == (k0 >> 5)) {
#pragma unroll
            for (int h = 1; h >= 0; --h) {
                const int l0 = (k0 & 31) + 8 * h, c = lane - l0;
                float r[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) r[q] = __shfl_sync(0xffffffffu, acc, l0 + q);
                if (c >= 0 && c < 8) {
                    const float *dc = Dv + (2 * b + h) * 64 + c;  // column c of the inverse, q >= c
                    float v = 0.f;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q >= c) v = fmaf(dc[q * 8], r[q], v);
                    acc = v;
                    xk[8 * h + c] = v;
                }
                if (h == 1) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) x[q] = __shfl_sync(0xffffffffu, acc, l0 + q);
                    if (et < k0 + 8) fold(k0 + 8, x);
                }
            }
        }
        gs.sync();
        if (et < k0) {
            if (w != (k0 >> 5)) {
                read8(xk + 8, x);
                fold(k0 + 8, x);
            }
            read8(xk, x);
            fold(k0, x);
        }
    }
}

}  // namespace als
