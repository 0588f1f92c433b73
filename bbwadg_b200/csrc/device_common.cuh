// Shared device-side definitions of the CUDA translation units.
#pragma once
#include <cuda_runtime.h>

#include "bbwadg.h"

namespace bbw {

#define NP(N) (((N) + 1) * ((N) + 2) * ((N) + 3) / 6)
#define NFP(N) (((N) + 1) * ((N) + 2) / 2)
// elements per CTA of the kernel-level entry points (256 threads)
#define VOL_EB(N) (512 / NP(N) > 0 ? 512 / NP(N) : 1)
#define SURF_EB(N) (512 / (4 * NFP(N)) > 0 ? 512 / (4 * NFP(N)) : 1)
#define UPD_EB(N) (256 / NP(N) > 0 ? 256 / NP(N) : 1)

// thread-local error record (errors.cu)
bbw_status set_error(bbw_status s, const char *msg);
bbw_status set_cuda_error(cudaError_t e, const char *where);
// checks the launch configuration error of the last kernel launch
bbw_status check_launch(const char *what);
// Raises `func`'s dynamic shared-memory limit on the current device to at
// least `bytes` (never lowers it).  The attribute is per kernel and per
// device, so it is tracked per (kernel, device); thread-safe; the CUDA
// status of the call is returned.
bbw_status ensure_smem_limit(const void *func, int bytes, const char *what);
template <class F>
inline bbw_status ensure_smem_limit(F *func, int bytes, const char *what) {
  return ensure_smem_limit(reinterpret_cast<const void *>(func), bytes, what);
}
// Launch of one stage kernel.  chained: the launch before it in the stream is
// another stage kernel, and this one may start before that has ended; it stages
// its constant operands and then waits for it (stage_wait), so launch latency
// and staging are hidden.  us per stage without / with: N = 1, K = 2058 4.9 / 4.1;
// N = 3, K = 384 7.8 / 7.0, K = 3072 10.3 / 9.4; N = 4, K = 3072 13.0 / 12.7; N = 5,
// K = 196608 417 / 411.  The coherent reads cost launches that are not chained
// nothing measurable: N = 8, K = 1296 188.5 / 188.7 single stages, N = 4, 8 taped
// shots of 24576 656 / 655.
template <class K, class P>
inline void launch_stage_kernel(K *kernel, int grid, int threads, size_t smem, cudaStream_t st,
                                bool chained, const P &params) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid), cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &a, cfg.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, params);
}
#ifdef __CUDACC__
// Waits until the stage before has ended and its writes are visible, then lets
// the next one start: every read of state, residual and clock comes after it
// and goes through the coherent path (no ld.global.nc: their pointers are not
// restrict-qualified, or the load says so), and at most two stages
// are ever in flight.  No-op in a launch that is not chained.
__device__ __forceinline__ void stage_wait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
#endif
// the device's opt-in maximum of dynamic shared memory per block (bytes)
int device_smem_optin();

}  // namespace bbw
