// sweep_fp32_p64.cu — FP32 half-sweep instances for f = 33..64 (sweep_fp32_tile.cuh).
#include "sweep_fp32_tile.cuh"

namespace als {

ALS_FP32_TILES(64) { return launch_tiles_of<64>(a, sp, st, launches); }

}  // namespace als
