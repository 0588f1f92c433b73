#include "ref_mma.cuh"
namespace bbw {
BBW_REF_RHS_INSTANCE(7)
}
