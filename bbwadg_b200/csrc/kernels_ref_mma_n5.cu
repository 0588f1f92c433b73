#include "ref_mma.cuh"
namespace bbw {
BBW_REF_RHS_INSTANCE(5)
BBW_REF_UPDATE_INSTANCE(5)
}
