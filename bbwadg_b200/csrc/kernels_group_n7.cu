#include "group_stage.cuh"
namespace bbw {
BBW_GROUP_STAGE_INSTANCE(7)
}
