// Host-visible description of a prepared warp-matrix stage launch
// (warp_stage.cuh, kernels_warp.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "bbwadg.h"

namespace bbw {

struct WarpPlan {
  bool on = false;       // the context may run its stage on this form
  bool pinned = false;   // chosen by the autotuner or the caller
  bool ops_sm = false;   // operators staged in shared memory
  int products = 4;      // products per split pair (4: FP32 contexts, 3: split FP16)
  int N = 0, K = 0, K0 = 0, Kc = 0, Nq = 0, bc = 0, S = 1, nsm = 148, max_ctas = 0;
  int pat_off = 0, table_ints = 0;
  int oDt = 0, oL = 0, oLt = 0, oV = 0, oVt = 0, oP = 0, ops_n = 0;
  float iD = 1.f, iL = 1.f, iV = 1.f, iP = 1.f, vnorm = 1.f;
  const float *geo = nullptr, *c2p = nullptr, *c2max = nullptr;
  const int *nbr = nullptr, *tables = nullptr;
  const uint4 *ops = nullptr;
  const int *src_tile = nullptr, *src_elem = nullptr;
  const float *src_vec = nullptr;
  float f0 = 0.f, tR = 0.f, samp = 0.f;
  const double *time = nullptr;
};

// Operators as FP16 pairs in the fragment order of the stage's B operands.
// Indices run in blocks of eight; a pair of blocks (16 nodes) interleaves so
// that one lane holds four consecutive nodes, an odd last block is in order
// (warp_node).  A k16 tile gives lane l (hi, hi, lo, lo) of operator row l/4
// and column pairs 2(l%4) of the pair's two blocks; a k8 tile (hi, lo).
// Order: D [3][KP][NB] and its k8 tiles [3][NB], LIFT [4][FP][NB] and [4][NB],
// Vq [chunk][KP][2] and [chunk][2], Pq [chunk][NB].  Sets the offsets, inverse
// scales and vnorm of the plan.
void warp_pack(WarpPlan &pl, const std::vector<float> *D, const std::vector<float> &LIFT,
               const std::vector<float> &Vq, const std::vector<float> &Pq,
               std::vector<uint32_t> &out);
bool warp_supported(int N);
// Whether the form is the default for `elements` (mesh elements times shots).
// A warp takes a 16-element tile from end to end, so a mesh of few tiles
// leaves most of the chip idle for the length of one tile, while the CTA-wide
// forms put 8 or 16 warps on a tile.  us per stage, this form against the FP32
// fused stage: N = 3, K = 3072: 11.5 / 10.2, K = 6000: 11.5 / 17.2; N = 5, K =
// 3072: 24.6 / 23.8, K = 6000: 25.4 / 43.1; N = 8, K = 1296: 206 / 187, K = 6000:
// 273 / 564.  At N = 6 and 7 it is the faster one from the smallest mesh on
// (K = 384: 44.7 / 73.3 and 80.4 / 112).
inline bool warp_preferred(int N, long long elements) {
  return N == 6 || N == 7 || elements > 296 * 16;
}
bbw_status warp_prepare(WarpPlan &pl);
bbw_status warp_launch(const WarpPlan &pl, const float *Qin, float *Qout, float *res, float fa,
                       float fb, float fdt, float cstage, cudaStream_t st);
// c2max[k] = max_q |c2q[k][q]|; c2p[k]: c2q[k] padded with zeros to a multiple of 16
bbw_status warp_medium(int K, int Nq, const float *c2q, float *c2max, float *c2p, cudaStream_t st);

}  // namespace bbw
