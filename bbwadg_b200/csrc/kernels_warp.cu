// Host side of the warp-matrix stage (warp_stage.cuh): operator packing,
// dispatch over N, per-element medium bounds.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "device_common.cuh"
#include "internal.h"
#include "warp_stage.h"

namespace bbw {

#define BBW_WARP_DECL(n)                                                                     \
  bbw_status warp_launch_##n(const WarpPlan &, const float *, float *, float *, float, float, \
                             float, float, cudaStream_t);                                    \
  bbw_status warp_prepare_##n(WarpPlan &);
BBW_WARP_DECL(1) BBW_WARP_DECL(2) BBW_WARP_DECL(3) BBW_WARP_DECL(4)
BBW_WARP_DECL(5) BBW_WARP_DECL(6) BBW_WARP_DECL(7) BBW_WARP_DECL(8)
#undef BBW_WARP_DECL

bool warp_supported(int N) { return N >= 1 && N <= 8; }

#define BBW_WARP_SWITCH(CALL)   \
  switch (N) {                  \
    case 1: CALL(1); break;     \
    case 2: CALL(2); break;     \
    case 3: CALL(3); break;     \
    case 4: CALL(4); break;     \
    case 5: CALL(5); break;     \
    case 6: CALL(6); break;     \
    case 7: CALL(7); break;     \
    case 8: CALL(8); break;     \
    default: return set_error(BBW_ERR_UNSUPPORTED, "warp-matrix stage: N out of range"); \
  }

bbw_status warp_launch(const WarpPlan &pl, const float *Qin, float *Qout, float *res, float fa,
                       float fb, float fdt, float cstage, cudaStream_t st) {
  const int N = pl.N;
#define CALL(n) return warp_launch_##n(pl, Qin, Qout, res, fa, fb, fdt, cstage, st)
  BBW_WARP_SWITCH(CALL)
#undef CALL
  return BBW_OK;
}

bbw_status warp_prepare(WarpPlan &pl) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  pl.nsm = nsm > 0 ? nsm : 148;
  const int N = pl.N;
#define CALL(n) return warp_prepare_##n(pl)
  BBW_WARP_SWITCH(CALL)
#undef CALL
  return BBW_OK;
}

// power of two that brings the largest |a| into [2^13, 2^14)
static float operator_scale(const float *a, size_t n) {
  float m = 0.f;
  for (size_t i = 0; i < n; ++i) m = std::max(m, std::fabs(a[i]));
  if (!(m > 0.f) || !std::isfinite(m)) return 1.f;
  int e = 0;
  std::frexp(m, &e);  // m in [2^(e-1), 2^e)
  return std::ldexp(1.f, std::min(std::max(14 - e, -100), 100));
}

static uint32_t pack_pair(float a, float b, bool lo) {
  const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
  uint16_t x, y;
  if (!lo) {
    x = __half_as_ushort(ha), y = __half_as_ushort(hb);
  } else {
    x = __half_as_ushort(__float2half_rn(a - __half2float(ha)));
    y = __half_as_ushort(__float2half_rn(b - __half2float(hb)));
  }
  return (uint32_t)x | (uint32_t)y << 16;
}

// index of slot c of block b when n indices are stored in blocks of eight
static int warp_node(int n, int b, int c) {
  const int nb = (n + 7) / 8;
  if (b == nb - 1 && nb % 2) return 8 * b + c;
  return 16 * (b / 2) + 4 * (c / 2) + 2 * (b % 2) + c % 2;
}

// tile of row block j and columns of pair (k16) or block (k8) k of the nr x nc
// column-major matrix A (row stride 1, column stride ld), zero outside
static void pack_tile(std::vector<uint32_t> &out, const float *A, int nr, int nc, int nrp, int ncp,
                      int ld, int j, int k, bool k16, float s) {
  for (int lane = 0; lane < 32; ++lane) {
    const int r = warp_node(nrp, j, lane / 4), c = 2 * (lane % 4);
    auto at = [&](int b, int slot) {
      const int col = warp_node(ncp, b, slot);
      return r < nr && col < nc ? A[r + (size_t)col * ld] * s : 0.f;
    };
    const int b0 = k16 ? 2 * k : k;
    for (int lo = 0; lo < 2; ++lo) {
      out.push_back(pack_pair(at(b0, c), at(b0, c + 1), lo));
      if (k16) out.push_back(pack_pair(at(b0 + 1, c), at(b0 + 1, c + 1), lo));
    }
  }
}

void warp_pack(WarpPlan &pl, const std::vector<float> *D, const std::vector<float> &LIFT,
               const std::vector<float> &Vq, const std::vector<float> &Pq,
               std::vector<uint32_t> &out) {
  const int N = pl.N, Np = np_of(N), Nfp = nfp_of(N), Nq = pl.Nq;
  const int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2, FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  const int nch = (Nq + 15) / 16, Nq16 = 16 * nch;
  float sD = operator_scale(D[0].data(), D[0].size());
  for (int d = 1; d < 3; ++d) sD = std::min(sD, operator_scale(D[d].data(), D[d].size()));
  const float sL = operator_scale(LIFT.data(), LIFT.size());
  const float sV = operator_scale(Vq.data(), Vq.size()), sP = operator_scale(Pq.data(), Pq.size());
  out.clear();
  auto at = [&]() { return (int)(out.size() / 4); };
  for (int d = 0; d < 3; ++d)
    for (int k = 0; k < KP; ++k)
      for (int j = 0; j < NB; ++j) pack_tile(out, D[d].data(), Np, Np, Np, Np, Np, j, k, true, sD);
  pl.oDt = at();
  for (int d = 0; d < 3 && KT; ++d)
    for (int j = 0; j < NB; ++j) pack_tile(out, D[d].data(), Np, Np, Np, Np, Np, j, 2 * KP, false, sD);
  pl.oL = at();
  auto face = [&](int f) { return LIFT.data() + (size_t)f * Nfp * Np; };
  for (int f = 0; f < 4; ++f)
    for (int k = 0; k < FP; ++k)
      for (int j = 0; j < NB; ++j) pack_tile(out, face(f), Np, Nfp, Np, Nfp, Np, j, k, true, sL);
  pl.oLt = at();
  for (int f = 0; f < 4 && FT; ++f)
    for (int j = 0; j < NB; ++j) pack_tile(out, face(f), Np, Nfp, Np, Nfp, Np, j, 2 * FP, false, sL);
  pl.oV = at();
  for (int c = 0; c < nch; ++c)
    for (int k = 0; k < KP; ++k)
      for (int h = 0; h < 2; ++h)
        pack_tile(out, Vq.data(), Nq, Np, Nq16, Np, Nq, 2 * c + h, k, true, sV);
  pl.oVt = at();
  for (int c = 0; c < nch && KT; ++c)
    for (int h = 0; h < 2; ++h)
      pack_tile(out, Vq.data(), Nq, Np, Nq16, Np, Nq, 2 * c + h, 2 * KP, false, sV);
  pl.oP = at();
  for (int c = 0; c < nch; ++c)
    for (int j = 0; j < NB; ++j) pack_tile(out, Pq.data(), Np, Nq, Np, Nq16, Np, j, c, true, sP);
  pl.ops_n = at();
  pl.iD = 1.f / sD, pl.iL = 1.f / sL, pl.iV = 1.f / sV, pl.iP = 1.f / sP;
  double vn = 0.0;
  for (int q = 0; q < Nq; ++q) {
    double s = 0.0;
    for (int n = 0; n < Np; ++n) s += std::fabs((double)Vq[q + (size_t)n * Nq]);
    vn = std::max(vn, s);
  }
  // twice the bound, as for the divergence: rounding cannot reach 2^16
  pl.vnorm = (float)(2.0 * vn);
}

// one warp per element
__global__ void k_medium(int K, int Nq, int Nq16, const float *__restrict__ c2q,
                         float *__restrict__ c2max, float *__restrict__ c2p) {
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= K) return;
  float m = 0.f;
  for (int q = lane; q < Nq16; q += 32) {
    const float v = q < Nq ? c2q[(size_t)k * Nq + q] : 0.f;
    m = fmaxf(m, fabsf(v));
    c2p[(size_t)k * Nq16 + q] = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) c2max[k] = m;
}

bbw_status warp_medium(int K, int Nq, const float *c2q, float *c2max, float *c2p,
                       cudaStream_t st) {
  k_medium<<<(K + 7) / 8, 256, 0, st>>>(K, Nq, (Nq + 15) / 16 * 16, c2q, c2max, c2p);
  return check_launch("medium bound");
}

}  // namespace bbw
