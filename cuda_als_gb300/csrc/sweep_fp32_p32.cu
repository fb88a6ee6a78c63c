// sweep_fp32_p32.cu — FP32 half-sweep instances for f <= 32 (sweep_fp32_tile.cuh).
#include "sweep_fp32_tile.cuh"

namespace als {

ALS_FP32_TILES(32) { return launch_tiles_of<32>(a, sp, st, launches); }

}  // namespace als
