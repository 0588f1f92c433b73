#include "ref_mma.cuh"
namespace bbw {
BBW_REF_UPDATE_INSTANCE(2)
}
