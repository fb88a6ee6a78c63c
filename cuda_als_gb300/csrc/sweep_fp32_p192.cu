// sweep_fp32_p192.cu — FP32 half-sweep instances for f = 129..175 (sweep_fp32_tile.cuh).
#include "sweep_fp32_tile.cuh"

namespace als {

ALS_FP32_TILES(192) { return launch_tiles_of<192>(a, sp, st, launches); }

}  // namespace als
