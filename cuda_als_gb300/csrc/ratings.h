// ratings.h — walking a row's ratings.  A row is the positions [beg, end) of the CSR, end up to
// INT32_MAX; walks that look ahead or step past `end` count in unsigned 32 bits, where the few
// thousand positions beyond do not wrap (in signed ones a row that ends within them of 2^31 - 1
// read far outside the array, or never ended).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ALS_HD __host__ __device__ __forceinline__
#else
#define ALS_HD inline
#endif

namespace als {

// Parts of `size` ratings that cover [at, end): none of an empty rest.
ALS_HD uint32_t parts_of(uint32_t at, uint32_t end, uint32_t size) {
    return (end - at + size - 1u) / size;
}
// Ratings of the part that starts at `at` <= end.
ALS_HD uint32_t part_ratings(uint32_t at, uint32_t end, uint32_t size) {
    return end - at < size ? end - at : size;
}
// Whether that part is the row's last.
ALS_HD bool part_is_last(uint32_t at, uint32_t end, uint32_t size) { return end - at <= size; }

}  // namespace als
