// index_kernels.cu — integer work of the sweep, bit-exact: stable LSD radix sorts, the stable
// CSR->CSC transpose and the degree order of rows.
//
// The reference transposes offline with scipy (data/netflix/prepare_netflix_data.py:102-109,
// data/toy_data_2/prepare_toy_data_2.py:195-200: R.tocsr(), R.tocsc()) and loads both layouts
// from disk (main.cpp:68-71).  Here the CSC is built on the GPU from the CSR: a stable sort of
// the entries by column index keeps them in row order inside each column, which is exactly the
// order scipy's csr_tocsc produces.  All of it is HBM-bound integer traffic: coalesced tiles of
// 4096 keys per CTA, one 256-bin histogram per tile, a scan of every digit's tile counts, then a
// stable scatter ranked with warp ballots.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "internal.h"

namespace als {

namespace {

constexpr int RADIX_BITS = 8;
constexpr int RADIX_BINS = 1 << RADIX_BITS;
constexpr int RADIX_THREADS = 256;  // histogram: a thread a bin
constexpr int RADIX_ROUNDS = 16;                          // keys a thread (histogram)
constexpr int RADIX_TILE = RADIX_THREADS * RADIX_ROUNDS;  // 4096
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
// The scatter is latency-bound (each CTA loads its whole tile, ranks it, then writes it): 512
// threads of 8 keys each, so that several CTAs of 16 warps fit an SM within its registers.
constexpr int SCAT_THREADS = 512;
constexpr int SCAT_WARPS = SCAT_THREADS / 32;                     // 16
constexpr int SCAT_ROUNDS = RADIX_TILE / SCAT_THREADS;            // 8 keys per lane
constexpr int SCAT_WARP_SPAN = 32 * SCAT_ROUNDS;                  // 256 contiguous keys / warp
static_assert(RADIX_TILE == TILE_KEYS && SCAT_WARP_SPAN <= 256 && SCAT_ROUNDS % 4 == 0, "tiles");
static_assert(SCAT_THREADS >= RADIX_BINS && RADIX_BINS % 32 == 0, "one thread per digit");

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
inline size_t array_bytes(int64_t n) { return align256(sizeof(int32_t) * (size_t)(n > 0 ? n : 1)); }
inline int64_t tiles_of(int64_t n) { return ceil_div(n > 0 ? n : 1, RADIX_TILE); }
inline int passes_of(int bits) { return std::max(1, (bits + RADIX_BITS - 1) / RADIX_BITS); }

// Exclusive scan, in place, of the `len` counts of row blockIdx.x; its total.
__global__ void __launch_bounds__(SCAN_THREADS)
scan_rows_kernel(int32_t *__restrict__ counts, int64_t len, int32_t *__restrict__ totals) {
    __shared__ int warp_sums[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *row = counts + (int64_t)blockIdx.x * len;
    int carry = 0;
    for (int64_t t0 = 0; t0 < len; t0 += SCAN_THREADS * SCAN_ITEMS) {
        const int64_t base = t0 + (int64_t)threadIdx.x * SCAN_ITEMS;
        int v[SCAN_ITEMS];
        int s = 0;
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i) {
            v[i] = base + i < len ? row[base + i] : 0;
            s += v[i];
        }
        int x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        int before = carry;
        for (int w = 0; w < SCAN_THREADS / 32; ++w) {
            const int y = warp_sums[w];
            before += w < warp ? y : 0;
            carry += y;
        }
        int pre = before + x - s;
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i) {
            if (base + i < len) row[base + i] = pre;
            pre += v[i];
        }
        __syncthreads();  // warp_sums is written again
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// ---- radix sort -----------------------------------------------------------------------------

__global__ void __launch_bounds__(RADIX_THREADS)
radix_hist_kernel(const uint32_t *__restrict__ keys, int64_t n, int shift, int64_t ntiles,
                  int32_t *__restrict__ hist) {
    __shared__ int h[RADIX_BINS];
    h[threadIdx.x] = 0;
    const int64_t base = (int64_t)blockIdx.x * RADIX_TILE;
    const int nvalid = (int)(n - base < RADIX_TILE ? n - base : RADIX_TILE);
    const uint32_t *k = keys + base;
    uint32_t d[RADIX_ROUNDS];
#pragma unroll
    for (int i = 0; i < RADIX_ROUNDS; ++i) {
        const int o = i * RADIX_THREADS + threadIdx.x;
        d[i] = o < nvalid ? k[o] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RADIX_ROUNDS; ++i)
        if (i * RADIX_THREADS + (int)threadIdx.x < nvalid)
            atomicAdd(&h[(d[i] >> shift) & (RADIX_BINS - 1)], 1);
    __syncthreads();
    hist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// What a scatter moves.
//   MOVE_PAIR    words `key` with a value each
//   MOVE_CSR     a transpose's first pass: the digit is column `key`'s lowest; the word that moves
//                on is the column's remaining bits above the row's `row_bits`, with a value
//   MOVE_TRIPLE  words `key` with two values each (`a`, `val`)
// A null `val` stands for the positions 0 .. n - 1.  Words and `a` are written through `keep`.
enum { MOVE_PAIR = 0, MOVE_CSR = 1, MOVE_TRIPLE = 2 };
struct Move {
    const uint32_t *key, *a, *val;  // a: MOVE_CSR rows, MOVE_TRIPLE the first value
    uint32_t *key_out, *a_out, *val_out;  // key_out: MOVE_TRIPLE only
    int shift;                      // the digit's place in the key
    int row_bits;                   // MOVE_CSR
    uint32_t high_mask;             // MOVE_CSR: bits of the column past its lowest digit
    uint32_t keep;
};

// Stable scatter.  Warp w of tile t owns the contiguous key range [t*4096 + w*256, +256) and
// walks it in 8 rounds of 32; a key's rank inside its warp is (keys of the same digit in earlier
// rounds) + (lanes below it with the same digit in this round), found with a ballot a digit bit.
// The warp offsets per digit are an exclusive prefix over warps on top of the tile's digit starts (a
// scan over digits).  The entries are first placed in shared memory in digit order (the tile sorted
// by digit), then streamed out: consecutive threads write consecutive addresses of a digit's run, so
// the global stores coalesce instead of scattering 32 ways per instruction.  hist: every digit's
// tile counts, scanned; totals: every digit's count (its start is scanned here).
// Shared memory sets the pace (random 8-byte stores, then rows of a digit), so a transpose moves
// two words a rating where they fit: 98.6M ratings into 17,770 columns 2.41 -> 1.55 ms (three words,
// sorted column ids kept for the pointers, scans of the whole histogram before), then 1.38 with
// ballots instead of match.any, values loaded behind the ranking and two CTAs an SM without spills
// instead of three (uniform columns: match.any 1.71, ballots 1.46, with three CTAs 1.58, with 1,024
// threads of four keys 1.61).
template <int MOVE>
__global__ void __launch_bounds__(SCAT_THREADS, 2)
radix_scatter_kernel(const Move mv, int64_t n, int64_t ntiles, const int32_t *__restrict__ hist,
                     const int32_t *__restrict__ totals) {
    extern __shared__ uint2 sorted[];  // [RADIX_TILE], then keys (TRIPLE) or digits (CSR)
    __shared__ int wcnt[SCAT_WARPS][RADIX_BINS];
    __shared__ int goff[RADIX_BINS];
    __shared__ int wsum[2][RADIX_BINS / 32];
    uint32_t *skey = reinterpret_cast<uint32_t *>(sorted + RADIX_TILE);
    uint8_t *sdig = reinterpret_cast<uint8_t *>(sorted + RADIX_TILE);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool digit_thread = tid < RADIX_BINS;  // whole warps: RADIX_BINS % 32 == 0
    // tile-local 32-bit offsets (n <= INT32_MAX): one 64-bit base per array
    const int64_t tile0 = (int64_t)blockIdx.x * RADIX_TILE;
    const int nvalid = (int)(n - tile0 < RADIX_TILE ? n - tile0 : RADIX_TILE);
    const int mine = warp * SCAT_WARP_SPAN + lane;  // this thread's first entry, then every 32nd
    const int left = nvalid - mine;
    uint32_t key[SCAT_ROUNDS], x[SCAT_ROUNDS], y[SCAT_ROUNDS];
    uint32_t rank[SCAT_ROUNDS / 4] = {};  // below SCAT_WARP_SPAN: four to a register
#pragma unroll
    for (int q = 0; q < SCAT_ROUNDS; ++q) {
        key[q] = 32 * q < left ? mv.key[tile0 + mine + 32 * q] : 0;
    }
    int first = 0, total = 0;
    if (digit_thread) {
        first = hist[(int64_t)tid * ntiles + blockIdx.x];
        total = totals[tid];
    }
    for (int i = tid; i < SCAT_WARPS * RADIX_BINS; i += SCAT_THREADS) (&wcnt[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < SCAT_ROUNDS; ++q) {
        const bool valid = 32 * q < left;
        const uint32_t d = (key[q] >> mv.shift) & (RADIX_BINS - 1);
        unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < RADIX_BITS; ++b) {
            const bool one = (d >> b) & 1;
            const unsigned m = __ballot_sync(0xffffffffu, one);
            peers &= one ? m : ~m;
        }
        const int before = valid ? wcnt[warp][d] : 0;
        rank[q / 4] |= (uint32_t)(before + __popc(peers & ((1u << lane) - 1u))) << 8 * (q % 4);
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) wcnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    // the rest of the entries is under way during the scans
#pragma unroll
    for (int q = 0; q < SCAT_ROUNDS; ++q) {
        const bool valid = 32 * q < left;
        x[q] = MOVE == MOVE_PAIR ? key[q] : valid ? mv.a[tile0 + mine + 32 * q] : 0;
        y[q] = !valid ? 0 : mv.val ? mv.val[tile0 + mine + 32 * q] : (uint32_t)(tile0 + mine + 32 * q);
    }
    __syncthreads();
    int cnt = 0, icnt = 0, itot = 0;  // keys of digit tid in this tile; inclusive scans over digits
    if (digit_thread) {
#pragma unroll 4
        for (int w = 0; w < SCAT_WARPS; ++w) cnt += wcnt[w][tid];
        icnt = cnt;
        itot = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, icnt, o), v = __shfl_up_sync(0xffffffffu, itot, o);
            if (lane >= o) {
                icnt += u;
                itot += v;
            }
        }
        if (lane == 31) {
            wsum[0][warp] = icnt;
            wsum[1][warp] = itot;
        }
    }
    __syncthreads();
    if (digit_thread) {
        int start = icnt - cnt, base = itot - total;
        for (int w = 0; w < warp; ++w) {
            start += wsum[0][w];
            base += wsum[1][w];
        }
        goff[tid] = base + first - start;  // a sorted slot j of digit d goes to goff[d] + j
#pragma unroll 4
        for (int w = 0; w < SCAT_WARPS; ++w) {
            const int t = wcnt[w][tid];
            wcnt[w][tid] = start;
            start += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < SCAT_ROUNDS; ++q) {
        if (32 * q >= left) continue;
        const uint32_t d = (key[q] >> mv.shift) & (RADIX_BINS - 1);
        const int lp = wcnt[warp][d] + (int)(rank[q / 4] >> 8 * (q % 4) & 0xffu);
        if (MOVE == MOVE_CSR) x[q] |= ((key[q] >> RADIX_BITS) & mv.high_mask) << mv.row_bits;
        sorted[lp] = make_uint2(x[q], y[q]);
        if (MOVE == MOVE_TRIPLE) skey[lp] = key[q];
        if (MOVE == MOVE_CSR) sdig[lp] = (uint8_t)d;
    }
    __syncthreads();
#pragma unroll 4
    for (int j = tid; j < nvalid; j += SCAT_THREADS) {
        const uint2 e = sorted[j];
        const uint32_t k = MOVE == MOVE_TRIPLE ? skey[j] : MOVE == MOVE_CSR ? sdig[j] : e.x;
        const uint32_t d = MOVE == MOVE_CSR ? k : (k >> mv.shift) & (RADIX_BINS - 1);
        const int dst = goff[d] + j;
        if (MOVE == MOVE_TRIPLE) mv.key_out[dst] = k;
        mv.a_out[dst] = e.x & mv.keep;
        mv.val_out[dst] = e.y;
    }
}

// The counters of a sort of n keys: [RADIX_BINS][tiles] tile counts and the digits' totals, two
// sets of the latter (a transpose needs those of its first pass after its last).
struct Counters {
    int32_t *hist, *totals[2];
};
inline size_t counter_bytes(int64_t n) {
    return align256(sizeof(int32_t) * RADIX_BINS * (size_t)tiles_of(n)) + 2 * sizeof(int32_t) * RADIX_BINS;
}
inline Counters counters_at(void *p, int64_t n) {
    Counters c;
    c.hist = (int32_t *)p;
    c.totals[0] = (int32_t *)((char *)p + align256(sizeof(int32_t) * RADIX_BINS * (size_t)tiles_of(n)));
    c.totals[1] = c.totals[0] + RADIX_BINS;
    return c;
}

// One pass: tile histograms, their scans, the scatter.  (The scatter's dynamic shared memory is
// raised first: static counters and tile together pass 48 KB.)
template <int MOVE>
cudaError_t radix_pass(const Move &mv, int64_t n, const Counters &c, int32_t *totals, cudaStream_t st) {
    const int64_t ntiles = tiles_of(n);
    const size_t dyn = RADIX_TILE * (sizeof(uint2) + (MOVE == MOVE_TRIPLE ? sizeof(uint32_t) : MOVE == MOVE_CSR ? 1 : 0));
    cudaError_t e = cudaFuncSetAttribute(radix_scatter_kernel<MOVE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    radix_hist_kernel<<<(unsigned)ntiles, RADIX_THREADS, 0, st>>>(mv.key, n, mv.shift, ntiles, c.hist);
    scan_rows_kernel<<<RADIX_BINS, SCAN_THREADS, 0, st>>>(c.hist, ntiles, totals);
    radix_scatter_kernel<MOVE><<<(unsigned)ntiles, SCAT_THREADS, dyn, st>>>(mv, n, ntiles, c.hist, totals);
    return cudaGetLastError();
}

// Row pointers are clamped to [0, nnz]: a malformed pointer array can never write outside.
__global__ void expand_rows_kernel(int64_t rows, int64_t nnz, const int32_t *__restrict__ ptr,
                                   int32_t *__restrict__ coo_rows) {
    const int lane = threadIdx.x & 31;
    int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = warp; r < rows; r += nwarps) {
        const int32_t b = max(0, min((int32_t)nnz, ptr[r])), e = max(b, min((int32_t)nnz, ptr[r + 1]));
        for (uint32_t k = b + lane; k < (uint32_t)e; k += 32) coo_rows[k] = (int32_t)r;
    }
}

// col_ptrs[c] = first position whose sorted key >= c (lower bound), written without atomics.
__global__ void col_ptrs_from_sorted_kernel(int64_t nnz, int64_t cols,
                                            const int32_t *__restrict__ skeys,
                                            int32_t *__restrict__ cptr) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p <= nnz;
         p += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = p == 0 ? 0 : (int64_t)skeys[p - 1] + 1;
        int64_t hi = p == nnz ? cols : (int64_t)skeys[p];
        lo = lo < 0 ? 0 : lo;  // keys outside [0, cols) cannot write outside cptr[0..cols]
        hi = hi > cols ? cols : hi;
        for (int64_t c = lo; c <= hi; ++c) cptr[c] = (int32_t)p;
    }
}

// Column pointers of a transpose by one or two passes, from its counters (scanned tile counts of
// the last pass, both passes' totals): with one, a column is a digit.  With two, the entries of
// columns (d1, d0) start, before the last pass, where those of the lowest digit d0 start
// (position s); column (d1, d0) starts where the pass sends the first entry of digit d1 at or
// after s: behind those of d1 in earlier tiles and in s's tile before s.  Block d0, a thread a d1.
__global__ void __launch_bounds__(RADIX_BINS)
col_ptrs_kernel(int passes, int64_t nnz, int64_t cols, int64_t ntiles, const uint32_t *__restrict__ words,
                int shift, const int32_t *__restrict__ hist, const int32_t *__restrict__ first_totals,
                const int32_t *__restrict__ last_totals, int32_t *__restrict__ cptr) {
    __shared__ int cnt[RADIX_BINS];
    __shared__ int wsum[2][RADIX_BINS / 32];
    __shared__ int start;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = first_totals[tid], t1 = last_totals[tid];
    int i0 = t0, i1 = t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, i0, o), v = __shfl_up_sync(0xffffffffu, i1, o);
        if (lane >= o) {
            i0 += u;
            i1 += v;
        }
    }
    if (lane == 31) {
        wsum[0][warp] = i0;
        wsum[1][warp] = i1;
    }
    cnt[tid] = 0;
    __syncthreads();
    int s0 = i0 - t0, s1 = i1 - t1;  // digit tid's start in the first and the last pass
    for (int w = 0; w < warp; ++w) {
        s0 += wsum[0][w];
        s1 += wsum[1][w];
    }
    if (blockIdx.x == 0 && tid == 0) cptr[cols] = (int32_t)nnz;
    if (passes == 1) {
        if (tid < cols) cptr[tid] = s0;
        return;
    }
    if (tid == (int)blockIdx.x) start = s0;
    __syncthreads();
    const int64_t t = start / RADIX_TILE;
    for (int64_t p = t * RADIX_TILE + tid; p < start; p += RADIX_BINS)
        atomicAdd(&cnt[(words[p] >> shift) & (RADIX_BINS - 1)], 1);
    __syncthreads();
    const int64_t c = ((int64_t)tid << RADIX_BITS) + blockIdx.x;
    if (c < cols) cptr[c] = s1 + (t < ntiles ? hist[tid * ntiles + t] + cnt[tid] : t1);
}

__global__ void degree_keys_kernel(int64_t rows, const int32_t *__restrict__ ptr, int32_t maxd,
                                   int32_t *__restrict__ keys) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (int64_t)gridDim.x * blockDim.x)
        keys[r] = maxd - (ptr[r + 1] - ptr[r]);
}

// Four entries a step, so that their loads overlap: 9.0M ratings 36.9 -> 16.0 us.
__global__ void count_bad_kernel(int64_t nnz, const int32_t *__restrict__ idx, int32_t limit,
                                 const float *__restrict__ val, int32_t *bad) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    int local = 0;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += 4 * step) {
        int32_t c[4];
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool on = p + q * step < nnz;
            c[q] = on ? idx[p + q * step] : 0;
            v[q] = on && val ? val[p + q * step] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (p + q * step < nnz && (c[q] < 0 || c[q] >= limit || !isfinite(v[q]))) ++local;
    }
    local = __reduce_add_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(bad, local);
}

int grid_for(int64_t work, int threads, int cap = 152 * 16) {
    int64_t g = ceil_div(work > 0 ? work : 1, threads);
    return (int)(g < cap ? g : cap);
}

}  // namespace

// ---------------------------------------------------------------------------------------------

size_t tile_counts_bytes(int64_t n) { return array_bytes(tiles_of(n)); }

cudaError_t scan_tile_counts(int32_t *counts, int64_t n, int32_t *total, cudaStream_t st) {
    scan_rows_kernel<<<1, SCAN_THREADS, 0, st>>>(counts, tiles_of(n), total);
    return cudaGetLastError();
}

size_t radix_sort_scratch_bytes(int64_t n, int values) {
    return (1 + (size_t)values) * array_bytes(n) + counter_bytes(n);
}

size_t radix_counter_bytes(int64_t n) { return counter_bytes(n); }

cudaError_t radix_sort_between(const int32_t *keys_in, const int32_t *vals_in,
                               int32_t *const (&set)[2][2], int64_t n, int bits, void *counters,
                               cudaStream_t st, int *last) {
    const Counters c = counters_at(counters, n);
    const int passes = passes_of(bits);
    *last = (passes - 1) & 1;
    if (n <= 0) return cudaSuccess;
    Move mv{};
    mv.key = (const uint32_t *)keys_in;
    mv.val = (const uint32_t *)vals_in;
    mv.keep = ~0u;
    for (int p = 0; p < passes; ++p) {
        mv.a_out = (uint32_t *)set[p & 1][0];
        mv.val_out = (uint32_t *)set[p & 1][1];
        mv.shift = p * RADIX_BITS;
        const cudaError_t e = radix_pass<MOVE_PAIR>(mv, n, c, c.totals[0], st);
        if (e != cudaSuccess) return e;
        mv.key = mv.a_out;
        mv.val = mv.val_out;
    }
    return cudaSuccess;
}

// The passes alternate between the scratch set and the outputs, so that the last one lands there.
cudaError_t radix_sort_pairs(const int32_t *keys_in, const int32_t *vals_in, int32_t *keys_out,
                             int32_t *vals_out, int64_t n, int bits, void *scratch,
                             cudaStream_t st) {
    int32_t *k2 = (int32_t *)scratch, *v2 = (int32_t *)((char *)scratch + array_bytes(n));
    void *counters = (char *)scratch + 2 * array_bytes(n);
    const bool odd = passes_of(bits) & 1;
    int32_t *const set[2][2] = {{odd ? keys_out : k2, odd ? vals_out : v2},
                                {odd ? k2 : keys_out, odd ? v2 : vals_out}};
    int last = 0;
    return radix_sort_between(keys_in, vals_in, set, n, bits, counters, st, &last);
}

cudaError_t radix_sort_triples(const int32_t *keys_in, const int32_t *a_in, const int32_t *b_in,
                               int32_t *keys_out, int32_t *a_out, int32_t *b_out, int64_t n,
                               int bits, void *scratch, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    char *s = (char *)scratch;
    const size_t arr = array_bytes(n);
    uint32_t *set[2][3] = {{(uint32_t *)keys_out, (uint32_t *)a_out, (uint32_t *)b_out},
                           {(uint32_t *)s, (uint32_t *)(s + arr), (uint32_t *)(s + 2 * arr)}};
    const Counters c = counters_at(s + 3 * arr, n);
    const int passes = passes_of(bits);
    Move mv{};
    mv.key = (const uint32_t *)keys_in;
    mv.a = (const uint32_t *)a_in;
    mv.val = (const uint32_t *)b_in;
    mv.keep = ~0u;
    for (int p = 0; p < passes; ++p) {
        uint32_t **dst = set[(passes - 1 - p) & 1];
        mv.key_out = dst[0];
        mv.a_out = dst[1];
        mv.val_out = dst[2];
        mv.shift = p * RADIX_BITS;
        const cudaError_t e = radix_pass<MOVE_TRIPLE>(mv, n, c, c.totals[0], st);
        if (e != cudaSuccess) return e;
        mv.key = dst[0];
        mv.a = dst[1];
        mv.val = dst[2];
    }
    return cudaSuccess;
}

// Whether one or two passes over packed words transpose the matrix: a word holds the row and what
// is left of the column after its lowest digit.
static bool transpose_packs(int64_t rows, int64_t cols) {
    const int cb = key_bits(cols);
    return cb <= 2 * RADIX_BITS && key_bits(rows) + std::max(0, cb - RADIX_BITS) <= 32;
}

// Two passes: a set of two words a rating (the rows of the CSR wait in the output's); one pass: the
// rows; the general path: the rows, a set of three words and the sorted columns.  And the counters.
// In place, the outputs are written in the last pass only: two passes keep the rows in scratch too,
// one pass takes copies of the columns and values.
static int transpose_arrays(int64_t rows, int64_t cols, bool in_place) {
    if (!transpose_packs(rows, cols)) return 5;
    return in_place ? 3 : passes_of(key_bits(cols)) == 2 ? 2 : 1;
}
size_t transpose_scratch_bytes(int64_t rows, int64_t cols, int64_t nnz, bool in_place) {
    return transpose_arrays(rows, cols, in_place) * array_bytes(nnz) + counter_bytes(nnz);
}

bool transposes_in_place(const als_csr_view &csr, const int32_t *ridx, const float *cval) {
    auto shares = [&](const void *out) {
        return share_words(out, csr.nnz, csr.col_idxs, csr.nnz) || share_words(out, csr.nnz, csr.vals, csr.nnz) ||
               share_words(out, csr.nnz, csr.row_ptrs, csr.rows + 1);
    };
    return csr.nnz > 0 && (shares(ridx) || shares(cval));
}

cudaError_t expand_rows(int64_t rows, int64_t nnz, const int32_t *ptr, int32_t *coo_rows,
                        cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    expand_rows_kernel<<<grid_for(rows * 32, 256), 256, 0, st>>>(rows, nnz, ptr, coo_rows);
    return cudaGetLastError();
}

cudaError_t csr_to_csc_device(int64_t rows, int64_t cols, int64_t nnz, const int32_t *ptr,
                              const int32_t *idx, const float *val, int32_t *cptr,
                              int32_t *ridx, float *cval, void *scratch, cudaStream_t st,
                              int32_t *coo_rows_out, int32_t *perm_out, bool rows_ready,
                              bool in_place) {
    if (nnz <= 0) return cudaMemsetAsync(cptr, 0, sizeof(int32_t) * (size_t)(cols + 1), st);
    const size_t arr = array_bytes(nnz);
    char *s = (char *)scratch;
    const int cb = key_bits(cols), rb = key_bits(rows), passes = passes_of(cb);
    const bool packs = transpose_packs(rows, cols), one = passes == 1;
    int32_t *coo_rows = coo_rows_out          ? coo_rows_out
                        : !packs || one       ? (int32_t *)s
                        : in_place            ? (int32_t *)(s + 2 * arr)
                                              : ridx;
    cudaError_t e = cudaSuccess;
    if (in_place && packs && one) {
        e = cudaMemcpyAsync(s + arr, idx, sizeof(int32_t) * (size_t)nnz, cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(s + 2 * arr, val, sizeof(float) * (size_t)nnz, cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return e;
        idx = (const int32_t *)(s + arr);
        val = (const float *)(s + 2 * arr);
    }
    if (!rows_ready) {
        e = expand_rows(rows, nnz, ptr, coo_rows, st);
        if (e != cudaSuccess) return e;
    }
    // the rating moves with its row, or its CSR position where the caller keeps the permutation
    const uint32_t *v_in = perm_out ? nullptr : (const uint32_t *)val;
    uint32_t *v_out = (uint32_t *)(perm_out ? perm_out : (int32_t *)cval);
    if (packs) {
        uint32_t *word = (uint32_t *)s, *pay = (uint32_t *)(s + arr);  // (two passes only)
        const Counters c = counters_at(s + transpose_arrays(rows, cols, in_place) * arr, nnz);
        Move mv{};
        mv.key = (const uint32_t *)idx;
        mv.a = (const uint32_t *)coo_rows;
        mv.val = v_in;
        mv.a_out = one ? (uint32_t *)ridx : word;
        mv.val_out = one ? v_out : pay;
        mv.row_bits = rb;
        mv.high_mask = one ? 0u : (1u << (cb - RADIX_BITS)) - 1u;
        mv.keep = ~0u;
        e = radix_pass<MOVE_CSR>(mv, nnz, c, c.totals[0], st);
        if (e != cudaSuccess) return e;
        if (!one) {
            mv.key = word;
            mv.val = pay;
            mv.a_out = (uint32_t *)ridx;
            mv.val_out = v_out;
            mv.shift = rb;
            mv.keep = (1u << rb) - 1u;
            e = radix_pass<MOVE_PAIR>(mv, nnz, c, c.totals[1], st);
            if (e != cudaSuccess) return e;
        }
        col_ptrs_kernel<<<one ? 1 : RADIX_BINS, RADIX_BINS, 0, st>>>(
            passes, nnz, cols, tiles_of(nnz), word, rb, c.hist, c.totals[0], c.totals[one ? 0 : 1], cptr);
    } else {
        int32_t *skeys = (int32_t *)(s + arr);
        // (an odd number of passes starts in the outputs: in place, one more over zero digits)
        const int bits = in_place && passes % 2 ? passes * RADIX_BITS + 1 : cb;
        e = radix_sort_triples(idx, coo_rows, (const int32_t *)v_in, skeys, ridx, (int32_t *)v_out,
                               nnz, bits, s + 2 * arr, st);
        if (e != cudaSuccess) return e;
        col_ptrs_from_sorted_kernel<<<grid_for(nnz + 1, 256), 256, 0, st>>>(nnz, cols, skeys, cptr);
    }
    if (perm_out) return gather_f32(nnz, perm_out, val, cval, st);
    return cudaGetLastError();
}

size_t degree_order_scratch_bytes(int64_t rows) {
    return 2 * array_bytes(rows) + radix_sort_scratch_bytes(rows, 1);
}

cudaError_t degree_order_device(int64_t rows, const int32_t *ptr, int32_t max_degree,
                                int32_t *perm, void *scratch, cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    const size_t arr = array_bytes(rows);
    char *s = (char *)scratch;
    int32_t *keys = (int32_t *)s;
    int32_t *skeys = (int32_t *)(s + arr);
    degree_keys_kernel<<<grid_for(rows, 256), 256, 0, st>>>(rows, ptr, max_degree, keys);
    return radix_sort_pairs(keys, nullptr, skeys, perm, rows, key_bits((int64_t)max_degree + 1), s + 2 * arr, st);
}

__global__ void gather_f32_kernel(int64_t n, const int32_t *__restrict__ perm,
                                  const float *__restrict__ src, float *__restrict__ dst) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x)
        dst[p] = src[perm[p]];
}

cudaError_t ptrs_from_sorted(int64_t n, int64_t nkeys, const int32_t *skeys, int32_t *ptr,
                             cudaStream_t st) {
    if (n <= 0) return cudaMemsetAsync(ptr, 0, sizeof(int32_t) * (size_t)(nkeys + 1), st);
    col_ptrs_from_sorted_kernel<<<grid_for(n + 1, 256), 256, 0, st>>>(n, nkeys, skeys, ptr);
    return cudaGetLastError();
}

cudaError_t gather_f32(int64_t n, const int32_t *perm, const float *src, float *dst,
                       cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    gather_f32_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, perm, src, dst);
    return cudaGetLastError();
}

cudaError_t count_bad_entries(int64_t nnz, const int32_t *idx, int32_t limit, const float *val,
                              int32_t *bad, cudaStream_t st) {
    if (nnz <= 0) return cudaSuccess;
    count_bad_kernel<<<grid_for(nnz, 4 * 256), 256, 0, st>>>(nnz, idx, limit, val, bad);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// CSR -> CSC without any allocation, for callers that may not allocate device memory.
//
// Some callers cannot call cudaMalloc (or have torch or any other allocator do it for them):
// plug-ins hosted by an engine that owns all device memory and forbids allocations inside its
// callbacks, and latency-critical loops that must not synchronise on the allocator.  For them the
// transpose's scratch lives in one file-scope device array of NOALLOC_SCRATCH_BYTES (16 MiB),
// which every GPU that loads this library holds until the process exits.  It admits
// NOALLOC_MAX_RATINGS (28 bytes a rating and 1 KiB of radix histograms per 4,096 ratings, of which
// the present transpose needs 20 at most); larger inputs are rejected with ALS_ERR_INVALID_ARG
// before anything runs.
//
// In host code the array's name is only a host-side stand-in, so the device address is looked up
// with cudaGetSymbolAddress (with the device current) on the first call made in each CUDA
// context, and looked up again when the device's context changes (after cudaDeviceReset the
// module reloads at another address).  Every call shares the one array, so each waits on the GPU for
// the one before, whatever its stream or thread: an event recorded behind every call (two calls
// that overlapped could take places from each other's counters, past the end of the outputs).  A call
// under stream capture is not ordered that way; replays of its graph must not overlap other calls.
// The transpose writes every scratch word before it reads it, so no clearing is needed between calls.
// ---------------------------------------------------------------------------------------------

namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = 16u << 20;
constexpr int64_t NOALLOC_MAX_RATINGS = 593856;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

// A device's array as one CUDA context sees it (an entry of a context that is gone never matches).
struct NoallocSite {
    unsigned long long ctx;  // cuCtxGetId; 0 where it is unavailable: looked up again each time
    void *addr;
    cudaEvent_t done;        // behind the last call's work (none without an id)
};
std::mutex g_noalloc_mu;
std::vector<NoallocSite> g_noalloc_sites[NOALLOC_MAX_DEVICES];

// The unique id of the calling thread's current CUDA context (cuCtxGetCurrent + cuCtxGetId
// through the runtime's driver entry points; no link against libcuda); 0 if unavailable.
unsigned long long current_context_id() {
    typedef int (*GetCurrentFn)(void **);
    typedef int (*GetIdFn)(void *, unsigned long long *);
    static const std::pair<GetCurrentFn, GetIdFn> fns = []() {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult qa = cudaDriverEntryPointSymbolNotFound, qb = qa;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &a, 12000, cudaEnableDefault, &qa) !=
                cudaSuccess || qa != cudaDriverEntryPointSuccess)
            a = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &b, 12000, cudaEnableDefault, &qb) !=
                cudaSuccess || qb != cudaDriverEntryPointSuccess)
            b = nullptr;
        return std::make_pair(reinterpret_cast<GetCurrentFn>(a), reinterpret_cast<GetIdFn>(b));
    }();
    void *ctx = nullptr;
    unsigned long long id = 0;
    if (!fns.first || !fns.second || fns.first(&ctx) != 0 || !ctx || fns.second(ctx, &id) != 0)
        return 0;
    return id;
}

}  // namespace

}  // namespace als

extern "C" als_status als_csr_to_csc_device_noalloc(const als_csr_view *csr, int32_t *col_ptrs,
                                                    int32_t *row_idxs, float *vals,
                                                    void *stream) {
    using namespace als;
    if (!csr || !col_ptrs || !csr->row_ptrs ||
        (csr->nnz > 0 && (!row_idxs || !vals || !csr->col_idxs || !csr->vals)))
        return set_global_error(ALS_ERR_INVALID_ARG, "null argument");
    if (csr->rows < 0 || csr->cols < 0 || csr->nnz < 0 || csr->nnz > INT32_MAX ||
        csr->rows >= INT32_MAX || csr->cols >= INT32_MAX)
        return set_global_error(ALS_ERR_INVALID_ARG, "shape out of range");
    const bool in_place = transposes_in_place(*csr, row_idxs, vals);
    if (csr->nnz > NOALLOC_MAX_RATINGS ||
        transpose_scratch_bytes(csr->rows, csr->cols, csr->nnz, in_place) > NOALLOC_SCRATCH_BYTES)
        return set_global_error(
            ALS_ERR_INVALID_ARG,
            "als_csr_to_csc_device_noalloc: " + std::to_string(csr->nnz) + " ratings, more than the " +
                std::to_string(NOALLOC_MAX_RATINGS) + " of its fixed " +
                std::to_string(NOALLOC_SCRATCH_BYTES) +
                "-byte scratch array; use als_csr_to_csc_device");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return set_global_error(ALS_ERR_NO_DEVICE, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES)
        return set_global_error(ALS_ERR_UNSUPPORTED, "device ordinal beyond 63");
    cudaStream_t st = (cudaStream_t)stream;
    // cudaGetDevice made the device's primary context current if it was not yet
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lock(g_noalloc_mu);  // until the call is enqueued
    NoallocSite site{0, nullptr, nullptr};
    for (const NoallocSite &k : g_noalloc_sites[dev])
        if (ctx != 0 && k.ctx == ctx) site = k;
    if (!site.addr) {  // set-up, once per device and context, with that device current
        e = cudaGetSymbolAddress(&site.addr, g_noalloc_scratch);
        if (e == cudaSuccess && ctx != 0) e = cudaEventCreateWithFlags(&site.done, cudaEventDisableTiming);
        if (e != cudaSuccess || !site.addr)
            return set_global_error(ALS_ERR_CUDA, std::string("the scratch array's address: ") +
                                                      cudaGetErrorString(e));
        site.ctx = ctx;
        if (ctx != 0) g_noalloc_sites[dev].push_back(site);
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const bool known = cudaStreamIsCapturing(st, &capture) == cudaSuccess;
    if (!known) cudaGetLastError();
    const bool ordered = site.done && known && capture == cudaStreamCaptureStatusNone;
    if (ordered) e = cudaStreamWaitEvent(st, site.done, 0);
    if (e == cudaSuccess)
        e = csr_to_csc_device(csr->rows, csr->cols, csr->nnz, csr->row_ptrs, csr->col_idxs,
                              csr->vals, col_ptrs, row_idxs, vals, site.addr, st, nullptr, nullptr,
                              false, in_place);
    // (behind whatever was enqueued, also when a later launch failed)
    if (ordered) {
        const cudaError_t r = cudaEventRecord(site.done, st);
        if (e == cudaSuccess) e = r;
    }
    if (e != cudaSuccess)
        return set_global_error(ALS_ERR_CUDA, std::string("csr_to_csc: ") + cudaGetErrorString(e));
    return ALS_OK;
}

