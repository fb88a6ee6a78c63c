// Walks rows that end at argv[1] with the helpers of ratings.h as the kernels do, and compares every
// part with 64-bit arithmetic.  Prints the parts checked.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "ratings.h"

using namespace als;

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    const int64_t end = std::atoll(argv[1]);
    long parts = 0;
    for (const int64_t size : {16, 32, 64, 128, 2048, 16384}) {
        for (int64_t degree = 0; degree <= 70000; degree += degree < 300 ? 1 : 997) {
            const int64_t beg = end - degree;
            // the kernels' walk: signed 32-bit bounds, unsigned positions
            const int32_t b32 = (int32_t)beg, e32 = (int32_t)end;
            if ((int64_t)parts_of(b32, e32, (uint32_t)size) != (degree + size - 1) / size) return 1;
            int64_t at = beg;
            for (uint32_t u = b32; u < (uint32_t)e32; u += (uint32_t)size, at += size, ++parts) {
                const int64_t want = end - at < size ? end - at : size;
                if ((int64_t)u != at || (int64_t)part_ratings(u, e32, (uint32_t)size) != want) return 1;
                if (part_is_last(u, e32, (uint32_t)size) != (at + size >= end)) return 1;
                // three parts ahead of this one, as the tiles' index loads look
                const uint32_t ahead = u + 3u * (uint32_t)size;
                if ((ahead < (uint32_t)e32) != (at + 3 * size < end)) return 1;
            }
            if (at < end) return 1;
            if (degree == 0 && (part_ratings(b32, e32, (uint32_t)size) != 0 || !part_is_last(b32, e32, (uint32_t)size)))
                return 1;
        }
    }
    std::printf("%ld\n", parts);
    return 0;
}
