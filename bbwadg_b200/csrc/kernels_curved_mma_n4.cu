#include "curved_mma.cuh"
namespace bbw {
BBW_CURVED_MMA_INSTANCE(4)
}
