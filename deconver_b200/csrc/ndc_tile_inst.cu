// The tile kernels for one storage type: compiled with -DNDC_TILE_T=0 (float32) and 1 (bfloat16).
#include "ndc_b200.h"
#include "ndc_common.cuh"
#include "ndc_tile.cuh"

#if NDC_TILE_T == 0
typedef float ndc_inst_t;
#else
typedef __nv_bfloat16 ndc_inst_t;
#endif

namespace ndc {
namespace tile {
NDC_TILE_INSTANCES(template, ndc_inst_t)
}  // namespace tile
}  // namespace ndc
