#include "warp_stage.cuh"
namespace bbw {
BBW_WARP_STAGE_INSTANCE(1)
}
