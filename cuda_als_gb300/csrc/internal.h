// internal.h — declarations shared by the translation units of libals_gb300 (not installed).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/als_gb300.h"

namespace als {

// Record a message for als_last_error(NULL) (thread-local) and return the status.
als_status set_global_error(als_status s, const std::string &msg);

#define ALS_TRY_CUDA(call, errvar)                                                           \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) {                                                             \
            errvar = std::string(#call) + ": " + cudaGetErrorString(e_);                     \
            return e_ == cudaErrorMemoryAllocation ? ALS_ERR_OUT_OF_MEMORY : ALS_ERR_CUDA;   \
        }                                                                                    \
    } while (0)

// ---------------------------------------------------------------------------------------------
// Index kernels (index_kernels.cu)
// ---------------------------------------------------------------------------------------------

// Significant bits of the keys 0 .. count - 1.
inline int key_bits(int64_t count) {
    int b = 0;
    while (b < 31 && (int64_t(1) << b) < count) ++b;
    return b;
}

// Bytes of scratch needed by a sort of n keys with `values` values each.
size_t radix_sort_scratch_bytes(int64_t n, int values);
// Stable LSD radix sorts of keys with one or two values each by the keys' lowest `bits` bits (at
// most 32; keys are unsigned).  A null last value stands for the positions 0..n-1.  Outputs may
// not be inputs; `scratch` holds radix_sort_scratch_bytes(n, values) bytes.
cudaError_t radix_sort_pairs(const int32_t *keys_in, const int32_t *vals_in, int32_t *keys_out,
                             int32_t *vals_out, int64_t n, int bits, void *scratch,
                             cudaStream_t st);
// The pairs' passes between two sets of (keys, values) of the caller's, the first into set[0];
// *last is the one that holds the result.  keys_in may be set[1]'s.  `counters` holds
// radix_counter_bytes(n) bytes.
size_t radix_counter_bytes(int64_t n);
cudaError_t radix_sort_between(const int32_t *keys_in, const int32_t *vals_in,
                               int32_t *const (&set)[2][2], int64_t n, int bits, void *counters,
                               cudaStream_t st, int *last);
cudaError_t radix_sort_triples(const int32_t *keys_in, const int32_t *a_in, const int32_t *b_in,
                               int32_t *keys_out, int32_t *a_out, int32_t *b_out, int64_t n,
                               int bits, void *scratch, cudaStream_t st);

// Counts per tile of TILE_KEYS keys: bytes for n keys, and their exclusive scan in place with the
// total in *total.
constexpr int TILE_KEYS = 4096;
size_t tile_counts_bytes(int64_t n);
cudaError_t scan_tile_counts(int32_t *counts, int64_t n, int32_t *total, cudaStream_t st);

// CSR -> CSC on the device, stable.  Scratch: transpose_scratch_bytes.  in_place: ridx or cval may
// share memory with the inputs (transposes_in_place).
size_t transpose_scratch_bytes(int64_t rows, int64_t cols, int64_t nnz, bool in_place = false);
bool transposes_in_place(const als_csr_view &csr, const int32_t *ridx, const float *cval);
cudaError_t csr_to_csc_device(int64_t rows, int64_t cols, int64_t nnz, const int32_t *ptr,
                              const int32_t *idx, const float *val, int32_t *cptr,
                              int32_t *ridx, float *cval, void *scratch, cudaStream_t st,
                              int32_t *coo_rows_out /* optional, nnz */,
                              int32_t *perm_out /* optional, nnz: CSC position -> CSR position */,
                              bool rows_ready = false /* coo_rows_out holds the rows already */,
                              bool in_place = false /* no coo_rows_out, no perm_out */);
// Host words to the device, there for whatever `st` runs next, `src` free to go.  (cudaMemcpy from
// pageable memory may return before the data has arrived, and a stream created non-blocking does
// not wait for it.)
inline cudaError_t upload(cudaStream_t st, int32_t *dst, const int32_t *src, size_t n) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, sizeof(int32_t) * n, cudaMemcpyHostToDevice, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}
// Whether n 32-bit words at a and k at b share memory.
inline bool share_words(const void *a, int64_t n, const void *b, int64_t k) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + 4 * (uintptr_t)k && y < x + 4 * (uintptr_t)n;
}

// ptr[k] = first position of the ascending keys skeys[0..n) that is >= k, for k in [0, nkeys]
// (the pointer array of sorted row or column indices).
cudaError_t ptrs_from_sorted(int64_t n, int64_t nkeys, const int32_t *skeys, int32_t *ptr,
                             cudaStream_t st);

// dst[p] = src[perm[p]]
cudaError_t gather_f32(int64_t n, const int32_t *perm, const float *src, float *dst,
                       cudaStream_t st);

// rows sorted by descending degree (stable).  Scratch: degree_order_scratch_bytes.
size_t degree_order_scratch_bytes(int64_t rows);
cudaError_t degree_order_device(int64_t rows, const int32_t *ptr, int32_t max_degree,
                                int32_t *perm, void *scratch, cudaStream_t st);

// The reference's srand(0) factor initialisation (als_model.cu:1772-1784) on the device: V gets
// 0.2 * rand() / RAND_MAX for its n f entries in order (glibc's sequence, bit for bit), U zeros.
cudaError_t init_factors_device(int64_t m, int64_t n, int f, float *U, float *V,
                                cudaStream_t st);

// Expand CSR row pointers into one row index per entry.
cudaError_t expand_rows(int64_t rows, int64_t nnz, const int32_t *ptr, int32_t *coo_rows,
                        cudaStream_t st);

// Validation: returns via *bad (device int) a nonzero count of entries with index outside
// [0, limit) or non-finite value.
cudaError_t count_bad_entries(int64_t nnz, const int32_t *idx, int32_t limit, const float *val,
                              int32_t *bad, cudaStream_t st);

// ---------------------------------------------------------------------------------------------
// Sweep kernels
// ---------------------------------------------------------------------------------------------

struct SweepArgs {
    const int32_t *ptr;     // rows + 1 (this side's CSR)
    const int32_t *idx;     // nnz, indices into the opposite table
    const float *val;       // nnz ratings
    const float *Y;         // opposite factors, FP32, row-contiguous (f per row)
    float *X;               // this side's factors (in: CG warm start, out: solution)
    const int32_t *order;   // row processing order (NULL = identity)
    int64_t nnz;            // ratings of the matrix
    int32_t row_begin;      // slice [row_begin, row_end) of the order
    int32_t row_end;
    int32_t f;
    float lambda;
    int32_t solve;          // ALS_SOLVE_*
    int32_t cg_iters;
    float cg_tol;
    int32_t *flags;         // [0] flagged rows (atomic), [1] fp64-refined rows
};

// Rows of the FP32 path heavier than FP32_SPLIT_RATINGS ratings: each split into parts of that
// many ratings whose partial Grams separate CTAs build, then added in order by one CTA per row
// that solves it.  The heavy rows are the first `nheavy` positions of the side's order.
constexpr int32_t FP32_SPLIT_RATINGS = 16384;
struct Fp32Split {
    const int32_t *part_beg = nullptr, *part_end = nullptr;  // device, per part
    const int32_t *first = nullptr;       // device, nheavy + 1: first part of each heavy row
    const int32_t *first_host = nullptr;  // host copy of `first`
    int32_t nheavy = 0;
    float *part = nullptr;                // parts x fp32_part_floats(f)
};
size_t fp32_part_floats(int f);

// Fused FP32 Gram + RHS + solve, one CTA per row (sweep_fp32.cu), heavy rows split.
bool fp32_supported(int f);
cudaError_t launch_sweep_fp32(const SweepArgs &a, const Fp32Split *sp, cudaStream_t st,
                              int *launches);

// ---------------------------------------------------------------------------------------------
// Evaluation (rmse.cu)
// ---------------------------------------------------------------------------------------------
size_t rmse_scratch_bytes();
// Deterministic FP64 sum of squared errors; writes the sum into *d_out (device double).
// sum over rows order[lo..hi) of ||A_r - B_r||^2 and ||A_r||^2 (FP64) into out[0..1]
cudaError_t launch_bucket_diff(const int32_t *order, int32_t lo, int32_t hi, const float *A,
                               const float *B, int f, double *out, cudaStream_t st);
cudaError_t launch_sq_error(int64_t nnz, const int32_t *rows, const int32_t *cols,
                            const float *vals, const float *U, const float *V, int f,
                            double *d_partials, double *d_out, cudaStream_t st);

}  // namespace als
