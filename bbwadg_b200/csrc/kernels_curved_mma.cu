// Host side of the curved matrix stage (curved_mma.cuh): dispatch over N and the
// point data of its tiles.
#include <cuda_runtime.h>

#include "curved.h"
#include "device_common.cuh"

namespace bbw {

#define BBW_DECL(n)                                                                             \
  bbw_status curved_mma_launch_##n(const CurvedMma &, const float *, float *, float *, cudaStream_t); \
  bbw_status curved_mma_prepare_##n(const CurvedMma &);
BBW_DECL(2) BBW_DECL(3) BBW_DECL(4) BBW_DECL(5)
#undef BBW_DECL

#define BBW_SWITCH(CALL) \
  switch (N) {           \
    case 2: CALL(2);     \
    case 3: CALL(3);     \
    case 4: CALL(4);     \
    case 5: CALL(5);     \
  }                      \
  return set_error(BBW_ERR_UNSUPPORTED, "curved matrix stage: N out of range");

bbw_status curved_mma_prepare(int N, CurvedMma &A) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  A.nsm = nsm > 0 ? nsm : 148;
#define CALL(n) return curved_mma_prepare_##n(A)
  BBW_SWITCH(CALL)
#undef CALL
}

bbw_status curved_mma_stage(int N, const CurvedMma &A, const float *Qold, float *Qnew, float *res,
                            cudaStream_t st) {
  if (A.KC == 0) return BBW_OK;
#define CALL(n) return curved_mma_launch_##n(A, Qold, Qnew, res, st)
  BBW_SWITCH(CALL)
#undef CALL
}

// src [KC][nc][n] -> dst [tile][c-major chunk of 16 points][nc][16 rows][16 points]; inv:
// reciprocals (0 past the data)
__global__ void k_tile_points(int KC, int nt, int nc, int n, int nch, int group, int slot, int ng,
                              bool inv, const float *__restrict__ src, float *__restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)nt * group * nch * nc * 256;
  if (i >= total) return;
  const int p = (int)(i & 15), row = (int)(i >> 4 & 15);
  long long j = i >> 8;
  const int c = (int)(j % nc);
  j /= nc;
  const int ch = (int)(j % nch);
  j /= nch;
  const int gr = (int)(j % group);
  const long long tile = j / group;
  const long long k = tile * 16 + row;
  const int q = 16 * ch + p;
  float v = 0.f;
  if (k < KC && q < n) {
    v = src[((k * group + gr) * nc + c) * n + q];
    if (inv) v = 1.f / v;
  }
  dst[((((tile * group + gr) * nch + ch) * ng + slot + c) * 16 + row) * 16 + p] = v;
}

// one warp per element
__global__ void k_curved_bounds(CurvedStageArgs S, float *__restrict__ bound) {
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= S.KC) return;
  float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int q = lane; q < S.Nq; q += 32) {
    const float J = fabsf(S.Jq[(size_t)k * S.Nq + q]);
    const float *g = S.vgeoq + (size_t)k * 9 * S.Nq + q;
    for (int c = 0; c < 3; ++c) {
      float a = 0.f, b = 0.f;
      for (int d = 0; d < 3; ++d) a += fabsf(g[(3 * c + d) * S.Nq]), b += fabsf(g[(3 * d + c) * S.Nq]);
      m[0] = fmaxf(m[0], a * J), m[1] = fmaxf(m[1], b * J);
    }
  }
  for (int q = lane; q < S.Nr; q += 32) {
    const float i = fabsf(1.f / S.Jr[(size_t)k * S.Nr + q]);
    m[2] = fmaxf(m[2], i * fabsf(S.c2q[(size_t)k * S.Nr + q])), m[3] = fmaxf(m[3], i);
  }
  for (int q = lane; q < 4 * S.Nfq; q += 32) {
    const int f = q / S.Nfq;
    const float s = fabsf(S.fgeoq[(((size_t)k * 4 + f) * 4 + 3) * S.Nfq + q - f * S.Nfq]);
    for (int j = 0; j < 4; ++j)
      if (j == f) m[4 + j] = fmaxf(m[4 + j], s);
  }
  for (int j = 0; j < 8; ++j) {
    for (int o = 16; o > 0; o >>= 1) m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
    if (lane == 0) bound[(size_t)k * 8 + j] = m[j];
  }
}

bbw_status curved_mma_points(const CurvedStageArgs &S, const CurvedMma &A, float *gq, float *fq,
                             float *jq, float *bound) {
  auto tiles = [&](int nc, int n, int nch, int group, int slot, int ng, bool inv, const float *src,
                   float *dst) {
    const long long total = (long long)A.nt * group * nch * nc * 256;
    k_tile_points<<<(int)((total + 255) / 256), 256>>>(S.KC, A.nt, nc, n, nch, group, slot, ng, inv,
                                                       src, dst);
  };
  tiles(9, S.Nq, A.nch, 1, 0, 10, false, S.vgeoq, gq);
  tiles(1, S.Nq, A.nch, 1, 9, 10, false, S.Jq, gq);
  tiles(4, S.Nfq, A.FC, 4, 0, 4, false, S.fgeoq, fq);
  tiles(1, S.Nr, A.nchr, 1, 0, 2, true, S.Jr, jq);
  tiles(1, S.Nr, A.nchr, 1, 1, 2, false, S.c2q, jq);
  k_curved_bounds<<<(S.KC + 7) / 8, 256>>>(S, bound);
  const bbw_status s = check_launch("curved point data");
  return s != BBW_OK ? s : set_cuda_error(cudaStreamSynchronize(nullptr), "curved point data");
}

}  // namespace bbw
