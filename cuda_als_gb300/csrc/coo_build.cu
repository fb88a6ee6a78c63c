// coo_build.cu — rating triples -> CSR (+ the row of every CSR entry) and CSC, on the GPU.
//
// The reference builds its input files offline with scipy: the raw (user, item, rating) triples
// of a split become coo_matrix((r, (u - 1, i - 1))), then .tocsr().tocoo() (entries in row-major
// order, duplicates summed), .tocsr() and .tocsc() (data/toy_data/prepare_toy_data.py:108-110,
// 147-150, 201-208; data/netflix/prepare_netflix_data.py:88-109), written as float32
// (.astype(np.float32)).  This is that step on the device:
//
//   1. stable LSD radix sort of the entries by (row, column) with their values: entries end in
//      that order, duplicates of a cell in input order.  Row and column share a 32-bit key where
//      they fit (8 bytes an entry and pass); otherwise the entries are sorted by column, then by
//      row, 12 bytes each;
//   2. a cell's first entry is its head: heads per tile and their scan give each cell's output
//      slot and the count after summing duplicates;
//   3. each head sums its cell's values in FP64, in input order, and rounds once to FP32.  scipy
//      sums the float64 (or integer) ratings before the float32 cast; an FP64 sum of float32
//      values on a common grid (star ratings) is exact, hence independent of order, so the
//      result is bit-identical to scipy's whenever that sum is exact (scipy's own per-row sort
//      is not stable, so no fixed order would do better).  The heads write the row pointers too;
//   4. the CSC by the library's stable transpose (rows ascending within a column: scipy's tocsc
//      order).
// 10.0M triples, 69,878 x 10,677: 2.80 -> 1.05 ms (positions sorted by column, then by row, with
// random gathers of rows, columns and values between, before).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "internal.h"

namespace als {

namespace {

inline size_t a256(size_t x) { return (x + 255) & ~size_t(255); }
inline int grid_of(int64_t work, int threads) {
    const int64_t g = (work + threads - 1) / threads;
    return (int)(g < 152 * 16 ? (g > 0 ? g : 1) : 152 * 16);
}

// Counts the triples with an index out of range; writes row << col_bits | column where `word` is
// given (rows and columns in range then fit 32 bits).  Four triples a step: their loads overlap.
__global__ void check_pack_kernel(int64_t nnz, const int32_t *__restrict__ r,
                                  const int32_t *__restrict__ c, int32_t rows, int32_t cols,
                                  int col_bits, uint32_t *__restrict__ word, int32_t *bad) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    int local = 0;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += 4 * step) {
        int32_t i[4], j[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool on = p + q * step < nnz;
            i[q] = on ? r[p + q * step] : 0;
            j[q] = on ? c[p + q * step] : 0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (p + q * step >= nnz) break;
            if (i[q] < 0 || i[q] >= rows || j[q] < 0 || j[q] >= cols) ++local;
            if (word) word[p + q * step] = (uint32_t)i[q] << col_bits | (uint32_t)j[q];
        }
    }
    local = __reduce_add_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(bad, local);
}

// The sorted entries: packed words (row null) or rows and columns.
struct Cells {
    const uint32_t *row, *word;
    const float *val;
    int col_bits;
    __device__ bool wide() const { return row != nullptr; }
    __device__ int32_t row_of(int64_t p) const { return (int32_t)(wide() ? row[p] : word[p] >> col_bits); }
    __device__ int32_t col_of(int64_t p) const {
        return (int32_t)(wide() ? word[p] : word[p] & ((1u << col_bits) - 1u));
    }
    __device__ bool same(int64_t p, int64_t q) const {
        return word[p] == word[q] && (!wide() || row[p] == row[q]);
    }
};

// A tile is TILE_KEYS entries: warp w's are [256 w, 256 w + 256), eight rounds of 32.  Bit q of
// the result: the thread's entry of round q is a head.
constexpr int CELL_THREADS = 512, CELL_ROUNDS = TILE_KEYS / CELL_THREADS;
__device__ __forceinline__ uint32_t heads_of(const Cells &c, int64_t first, int64_t n) {
    uint32_t heads = 0;
#pragma unroll
    for (int q = 0; q < CELL_ROUNDS; ++q) {
        const int64_t p = first + 32 * q;
        if (p < n && (p == 0 || !c.same(p, p - 1))) heads |= 1u << q;
    }
    return heads;
}
__device__ __forceinline__ int64_t first_entry() {
    return (int64_t)blockIdx.x * TILE_KEYS + (threadIdx.x >> 5) * 32 * CELL_ROUNDS + (threadIdx.x & 31);
}

__global__ void __launch_bounds__(CELL_THREADS)
count_heads_kernel(const Cells c, int64_t n, int32_t *__restrict__ counts) {
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    const int k = __reduce_add_sync(0xffffffffu, __popc(heads_of(c, first_entry(), n)));
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, k);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// Each cell's head writes the cell: its row, column and the FP64 sum of its values in input
// order, rounded once to FP32; and the pointers of the rows that start with it.
__global__ void __launch_bounds__(CELL_THREADS)
emit_kernel(const Cells c, int64_t n, int64_t rows, const int32_t *__restrict__ slots,
            const int32_t *__restrict__ cells, int32_t *__restrict__ row_ptrs,
            int32_t *__restrict__ out_row, int32_t *__restrict__ out_col,
            float *__restrict__ out_val) {
    __shared__ int wsum[CELL_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t first = first_entry();
    const uint32_t heads = heads_of(c, first, n);
    const int mine = __reduce_add_sync(0xffffffffu, __popc(heads));
    if (lane == 0) wsum[warp] = mine;
    __syncthreads();
    int k = slots[blockIdx.x];
    for (int w = 0; w < warp; ++w) k += wsum[w];
#pragma unroll
    for (int q = 0; q < CELL_ROUNDS; ++q) {
        const int64_t p = first + 32 * q;
        const bool head = (heads >> q) & 1;
        const unsigned m = __ballot_sync(0xffffffffu, head);
        if (p < n) {
            const int32_t r = c.row_of(p);
            if (head) {
                const int slot = k + __popc(m & ((1u << lane) - 1u));
                double s = (double)c.val[p];
                for (int64_t t = p + 1; t < n && c.same(t, p); ++t) s += (double)c.val[t];
                if (out_row) out_row[slot] = r;
                out_col[slot] = c.col_of(p);
                out_val[slot] = (float)s;
                for (int64_t i = p == 0 ? 0 : (int64_t)c.row_of(p - 1) + 1; i <= r; ++i)
                    row_ptrs[i] = slot;
            }
            if (p == n - 1)
                for (int64_t i = (int64_t)r + 1; i <= rows; ++i) row_ptrs[i] = *cells;
        }
        k += __popc(m);
    }
}

}  // namespace

// Whether row and column share a 32-bit key.
static bool coo_packs(int64_t rows, int64_t cols) { return key_bits(rows) + key_bits(cols) <= 32; }

// Whether the CSC's arrays can hold entries between passes: not where they share memory with the
// values, which the first pass reads (rows and columns are packed before it).
static bool sorts_in_csc(int64_t nnz, const float *val, const int32_t *csc_rows,
                         const float *csc_vals) {
    return csc_rows && !share_words(csc_rows, nnz, val, nnz) && !share_words(csc_vals, nnz, val, nnz);
}

// Flags and heads per tile; then the sort's entries and counters, of which the transpose takes the
// place.  Packed, the entries pass between one set of two words here and the arrays of the CSC
// (scratch has to be mapped on every call: 0.34 ms of 1.44 for five arrays of 10.0M entries), or a
// second set here.
size_t coo_build_scratch_bytes(int64_t rows, int64_t cols, int64_t nnz, bool csc, bool in_csc) {
    const size_t arr = a256(sizeof(int32_t) * (size_t)(nnz > 0 ? nnz : 1));
    const size_t sort = coo_packs(rows, cols) ? (in_csc ? 2 : 4) * arr + radix_counter_bytes(nnz)
                                              : 6 * arr + radix_sort_scratch_bytes(nnz, 2);
    return 256 + a256(tile_counts_bytes(nnz)) +
           std::max(sort, csc ? transpose_scratch_bytes(rows, cols, nnz) : 0);
}

// Device core.  `*nnz_out` (host) receives the cell count; the stream is synchronised to read the
// validation count, to read the cell count (every later launch depends on them) and at the end.
// *bad_out receives the number of triples with an index outside [0, rows) x [0, cols); then
// nothing is built.
cudaError_t coo_to_csr_device(int64_t rows, int64_t cols, int64_t nnz, const int32_t *ridx,
                              const int32_t *cidx, const float *val, int32_t *row_ptrs,
                              int32_t *col_idxs, float *vals, int32_t *coo_rows,
                              int32_t *col_ptrs, int32_t *csc_rows, float *csc_vals,
                              void *scratch, cudaStream_t st, int64_t *nnz_out, int *bad_out) {
    *nnz_out = 0;
    *bad_out = 0;
    if (nnz <= 0) {
        cudaError_t e = cudaMemsetAsync(row_ptrs, 0, sizeof(int32_t) * (size_t)(rows + 1), st);
        if (e == cudaSuccess && col_ptrs)
            e = cudaMemsetAsync(col_ptrs, 0, sizeof(int32_t) * (size_t)(cols + 1), st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        return e;
    }
    const size_t arr = a256(sizeof(int32_t) * (size_t)nnz);
    char *s = (char *)scratch;
    int32_t *flags = (int32_t *)s;  // [0] bad triples, [1] cells
    s += 256;
    int32_t *counts = (int32_t *)s;
    s += a256(tile_counts_bytes(nnz));
    void *tail = s;
    const int rb = key_bits(rows), cb = key_bits(cols);
    const bool packed = coo_packs(rows, cols);
    auto array = [&](int k) { return (int32_t *)(s + k * arr); };

    cudaError_t e = cudaMemsetAsync(flags, 0, 2 * sizeof(int32_t), st);
    if (e != cudaSuccess) return e;
    check_pack_kernel<<<grid_of(nnz, 4 * 256), 256, 0, st>>>(nnz, ridx, cidx, (int32_t)rows,
                                                             (int32_t)cols, cb,
                                                             packed ? (uint32_t *)array(0) : nullptr,
                                                             flags);
    int32_t got = 0;
    e = cudaMemcpyAsync(&got, flags, sizeof(got), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    if (got) {
        *bad_out = got;
        return cudaSuccess;
    }
    // 1. by row and column
    Cells c{};
    c.col_bits = cb;
    if (packed) {
        const bool in_csc = sorts_in_csc(nnz, val, csc_rows, csc_vals);
        int32_t *const set[2][2] = {{in_csc ? csc_rows : array(2), in_csc ? (int32_t *)csc_vals : array(3)},
                                    {array(0), array(1)}};
        int last = 0;
        e = radix_sort_between(array(0), (const int32_t *)val, set, nnz, rb + cb, array(in_csc ? 2 : 4), st,
                               &last);
        c.word = (const uint32_t *)set[last][0];
        c.val = (const float *)set[last][1];
    } else {
        e = radix_sort_triples(cidx, ridx, (const int32_t *)val, array(0), array(1), array(2), nnz, cb,
                               array(6), st);
        if (e == cudaSuccess)
            e = radix_sort_triples(array(1), array(0), array(2), array(3), array(4), array(5), nnz, rb,
                                   array(6), st);
        c.row = (const uint32_t *)array(3);
        c.word = (const uint32_t *)array(4);
        c.val = (const float *)array(5);
    }
    if (e != cudaSuccess) return e;
    // 2. cells and their slots
    const unsigned ntiles = (unsigned)((nnz + TILE_KEYS - 1) / TILE_KEYS);
    count_heads_kernel<<<ntiles, CELL_THREADS, 0, st>>>(c, nnz, counts);
    e = scan_tile_counts(counts, nnz, flags + 1, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(&got, flags + 1, sizeof(got), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    const int64_t cells = got;
    // 3. one entry per cell, duplicates summed
    emit_kernel<<<ntiles, CELL_THREADS, 0, st>>>(c, nnz, rows, counts, flags + 1, row_ptrs, coo_rows,
                                                 col_idxs, vals);
    // 4. the CSC
    e = cudaGetLastError();
    if (e == cudaSuccess && col_ptrs)
        e = csr_to_csc_device(rows, cols, cells, row_ptrs, col_idxs, vals, col_ptrs, csc_rows,
                              csc_vals, tail, st, coo_rows, nullptr, coo_rows != nullptr);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(st);
    *nnz_out = cells;
    return e;
}

}  // namespace als

using namespace als;

static als_status coo_args(const als_coo_view *coo, const int32_t *row_ptrs,
                           const int32_t *col_idxs, const float *vals, const int32_t *col_ptrs,
                           const int32_t *csc_rows, const float *csc_vals,
                           const int64_t *nnz_out) {
    if (!coo || !row_ptrs || !nnz_out)
        return set_global_error(ALS_ERR_INVALID_ARG, "null argument");
    if (coo->nnz > 0 && (!coo->row_idxs || !coo->col_idxs || !coo->vals || !col_idxs || !vals))
        return set_global_error(ALS_ERR_INVALID_ARG, "null array");
    if (!!col_ptrs != !!csc_rows || !!col_ptrs != !!csc_vals)
        return set_global_error(ALS_ERR_INVALID_ARG,
                                "col_ptrs, row_idxs and csc_vals: all three or none");
    if (coo->rows < 0 || coo->cols < 0 || coo->nnz < 0 || coo->nnz > INT32_MAX ||
        coo->rows >= INT32_MAX || coo->cols >= INT32_MAX)
        return set_global_error(ALS_ERR_INVALID_ARG, "shape out of range");
    return ALS_OK;
}

static als_status cuda_fail(const char *what, cudaError_t e) {
    return set_global_error(e == cudaErrorMemoryAllocation ? ALS_ERR_OUT_OF_MEMORY : ALS_ERR_CUDA,
                            std::string(what) + ": " + cudaGetErrorString(e));
}

static als_status bad_index(int bad) {
    return set_global_error(ALS_ERR_INVALID_ARG,
                            std::to_string(bad) + " triples with a row or column index out of range");
}

extern "C" als_status als_coo_to_csr_device(const als_coo_view *coo, int32_t *row_ptrs,
                                            int32_t *col_idxs, float *vals, int32_t *coo_rows,
                                            int32_t *col_ptrs, int32_t *row_idxs,
                                            float *csc_vals, int64_t *nnz_out, void *stream) {
    als_status s = coo_args(coo, row_ptrs, col_idxs, vals, col_ptrs, row_idxs, csc_vals, nnz_out);
    if (s != ALS_OK) return s;
    cudaStream_t st = (cudaStream_t)stream;
    void *scratch = nullptr;
    const bool in_csc = sorts_in_csc(coo->nnz, coo->vals, row_idxs, csc_vals);
    cudaError_t e = cudaMallocAsync(&scratch, coo_build_scratch_bytes(coo->rows, coo->cols, coo->nnz,
                                                                      col_ptrs != nullptr, in_csc), st);
    if (e != cudaSuccess) return cuda_fail("cudaMallocAsync", e);
    int bad = 0;
    e = coo_to_csr_device(coo->rows, coo->cols, coo->nnz, coo->row_idxs, coo->col_idxs,
                          coo->vals, row_ptrs, col_idxs, vals, coo_rows, col_ptrs, row_idxs,
                          csc_vals, scratch, st, nnz_out, &bad);
    cudaFreeAsync(scratch, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail("coo_to_csr", e);
    if (bad) return bad_index(bad);
    return ALS_OK;
}

extern "C" als_status als_coo_to_csr(const als_coo_view *coo, int32_t *row_ptrs,
                                     int32_t *col_idxs, float *vals, int32_t *coo_rows,
                                     int32_t *col_ptrs, int32_t *row_idxs, float *csc_vals,
                                     int64_t *nnz_out) {
    als_status s = coo_args(coo, row_ptrs, col_idxs, vals, col_ptrs, row_idxs, csc_vals, nnz_out);
    if (s != ALS_OK) return s;
    *nnz_out = 0;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return set_global_error(ALS_ERR_NO_DEVICE, "no CUDA device");
    const int64_t rows = coo->rows, cols = coo->cols, nnz = coo->nnz;
    const size_t n4 = sizeof(int32_t) * (size_t)(nnz > 0 ? nnz : 1);
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return cuda_fail("cudaStreamCreate", e);
    char *buf = nullptr;
    // inputs (3 nnz), CSR (rows + 1, 2 nnz), COO rows (nnz), CSC (cols + 1, 2 nnz), scratch
    const size_t a_in = 3 * a256(n4), a_csr = a256(sizeof(int32_t) * (rows + 1)) + 2 * a256(n4);
    const size_t a_rows = a256(n4), a_csc = a256(sizeof(int32_t) * (cols + 1)) + 2 * a256(n4);
    const size_t a_scr = coo_build_scratch_bytes(rows, cols, nnz, col_ptrs != nullptr, col_ptrs != nullptr);
    e = cudaMalloc(&buf, a_in + a_csr + a_rows + a_csc + a_scr);
    if (e != cudaSuccess) {
        cudaStreamDestroy(st);
        return cuda_fail("cudaMalloc", e);
    }
    char *q = buf;
    int32_t *d_r = (int32_t *)q; q += a256(n4);
    int32_t *d_c = (int32_t *)q; q += a256(n4);
    float *d_v = (float *)q; q += a256(n4);
    int32_t *d_ptr = (int32_t *)q; q += a256(sizeof(int32_t) * (rows + 1));
    int32_t *d_idx = (int32_t *)q; q += a256(n4);
    float *d_val = (float *)q; q += a256(n4);
    int32_t *d_rows = (int32_t *)q; q += a256(n4);
    int32_t *d_cptr = (int32_t *)q; q += a256(sizeof(int32_t) * (cols + 1));
    int32_t *d_ridx = (int32_t *)q; q += a256(n4);
    float *d_cval = (float *)q; q += a256(n4);
    void *d_scr = q;
    auto step = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    if (nnz > 0) {
        step(cudaMemcpyAsync(d_r, coo->row_idxs, n4, cudaMemcpyHostToDevice, st));
        step(cudaMemcpyAsync(d_c, coo->col_idxs, n4, cudaMemcpyHostToDevice, st));
        step(cudaMemcpyAsync(d_v, coo->vals, n4, cudaMemcpyHostToDevice, st));
    }
    int bad = 0;
    if (e == cudaSuccess)
        e = coo_to_csr_device(rows, cols, nnz, d_r, d_c, d_v, d_ptr, d_idx, d_val,
                              coo_rows ? d_rows : nullptr, col_ptrs ? d_cptr : nullptr,
                              col_ptrs ? d_ridx : nullptr, col_ptrs ? d_cval : nullptr, d_scr, st,
                              nnz_out, &bad);
    const size_t k4 = sizeof(int32_t) * (size_t)*nnz_out;
    if (e == cudaSuccess && !bad) {
        step(cudaMemcpyAsync(row_ptrs, d_ptr, sizeof(int32_t) * (rows + 1), cudaMemcpyDeviceToHost, st));
        if (k4) {
            step(cudaMemcpyAsync(col_idxs, d_idx, k4, cudaMemcpyDeviceToHost, st));
            step(cudaMemcpyAsync(vals, d_val, k4, cudaMemcpyDeviceToHost, st));
            if (coo_rows) step(cudaMemcpyAsync(coo_rows, d_rows, k4, cudaMemcpyDeviceToHost, st));
        }
        if (col_ptrs) {
            step(cudaMemcpyAsync(col_ptrs, d_cptr, sizeof(int32_t) * (cols + 1), cudaMemcpyDeviceToHost, st));
            if (k4) {
                step(cudaMemcpyAsync(row_idxs, d_ridx, k4, cudaMemcpyDeviceToHost, st));
                step(cudaMemcpyAsync(csc_vals, d_cval, k4, cudaMemcpyDeviceToHost, st));
            }
        }
        step(cudaStreamSynchronize(st));
    }
    cudaStreamSynchronize(st);
    cudaFree(buf);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) return cuda_fail("coo_to_csr", e);
    if (bad) return bad_index(bad);
    return ALS_OK;
}
