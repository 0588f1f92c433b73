// Matrix forms of the kernel-level entry points (ref_mma.cuh), by N.
#pragma once
#include <cuda_runtime.h>

#include "bbwadg.h"

namespace bbw {

#define BBW_REF_RHS_DECL(n)                                                                      \
  bbw_status ref_volume_##n(int, const float *, const float *, const float *, const float *,     \
                            const float *, float *, cudaStream_t);                               \
  bbw_status ref_surface_##n(int, int, const float *, const int *, const int *, const float *,   \
                             const float *, float *, cudaStream_t);
#define BBW_REF_UPDATE_DECL(n)                                                                   \
  bool ref_update_fits_##n(int Nq);                                                              \
  bbw_status ref_update_##n(int, int, const float *, const float *, const float *, const float *, \
                            float, float, float, const float *, float *, float *, cudaStream_t);
BBW_REF_RHS_DECL(3) BBW_REF_RHS_DECL(4) BBW_REF_RHS_DECL(5) BBW_REF_RHS_DECL(6) BBW_REF_RHS_DECL(7)
BBW_REF_UPDATE_DECL(3) BBW_REF_UPDATE_DECL(4) BBW_REF_UPDATE_DECL(5) BBW_REF_UPDATE_DECL(6)
#undef BBW_REF_RHS_DECL
#undef BBW_REF_UPDATE_DECL

}  // namespace bbw
