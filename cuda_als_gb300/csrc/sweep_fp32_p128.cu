// sweep_fp32_p128.cu — FP32 half-sweep instances for f = 65..128 (sweep_fp32_tile.cuh).
#include "sweep_fp32_tile.cuh"

namespace als {

ALS_FP32_TILES(128) { return launch_tiles_of<128>(a, sp, st, launches); }

}  // namespace als
