// Internal interface of the fused curved-element stage (kernels_curved.cu),
// used by the curvilinear solver handle (capi_curved.cu).
#pragma once
#include <cuda_runtime.h>

#include "bbwadg.h"

namespace bbw {

// One LSRK stage of the curved elements k = k_off + i, i < KC.  Geometry rows
// are compact (row i): vgeoq [KC][9][Nq], Jq [KC][Nq], fgeoq [KC][4][4][Nfq],
// Jr / c2q [KC][Nr] at the update's cubature.  Operators column-major as the
// reference uploads them; vmapP [K][4Nfp] in the handle's element order.
struct CurvedStageArgs {
  int KC, k_off, Nq, Nfq, Nr, EB;
  const float *vgeoq, *Jq, *fgeoq, *Jr, *c2q;
  const float *Vq, *Vrq, *Vsq, *Vtq, *Pq, *Prq, *Psq, *Ptq, *VfqFace, *Pfq, *Vqr, *Pqr;
  const int *Fmask, *vmapP;
  float fa, fb, fdt;
};

// reads Qold (own element and neighbour traces), writes Qnew and res of the
// KC curved elements
bbw_status curved_stage(int N, const CurvedStageArgs &A, const float *Qold, float *Qnew,
                        float *res, cudaStream_t st);

// The same stage on warp-level matrix instructions (curved_mma.cuh): operators as
// split tiles (warp_stage.h), point data of 16-element tiles in the order the
// lanes read it, [row][16 points] per quantity and chunk of 16 points, zero past
// the rule: gq [nt][nch][10] (vgeoq 9, J), fq [nt][4][FC][4] (nx ny nz sJ), jq
// [nt][nchr][2] (1/J, c2).  bound [KC][8]: largest sum_d |J g_cd|, sum_c |J g_cd|,
// c2/J, 1/J, and sJ of the four faces.
struct CurvedMma {
  bool on = false;
  int KC = 0, k_off = 0, nt = 0, nch = 0, nchr = 0, FC = 0, nsm = 148, scratch = 0;
  int oV[4] = {}, oVt[4] = {}, oP[4] = {};  // Vq Vrq Vsq Vtq, k8 tails, Pq Prq Psq Ptq
  int oF = 0, oFt = 0, oL = 0;              // VfqFace, Pfq by face and chunk
  int oVr = 0, oVrt = 0, oPr = 0;           // update's Vq, Pq
  int oM = 0;                               // plane of the rests
  float iV = 1.f, iD = 1.f, iP = 1.f, iF = 1.f, iVr = 1.f, iPr = 1.f;  // inverse scales
  float vnorm = 1.f, dnorm = 1.f, fnorm = 1.f, rnorm = 1.f;            // row sums
  float fa = 0.f, fb = 0.f, fdt = 0.f;
  const uint4 *ops = nullptr;
  const float *gq = nullptr, *fq = nullptr, *jq = nullptr, *bound = nullptr;
  const int *Fmask = nullptr, *vmapP = nullptr;
};
// Whether the matrix form is the faster one for KC curved elements: its tile
// is a longer chain than the thread-per-output kernel's block, so it wants
// enough tiles.  us per stage with the planar elements beside them, thread per
// output / matrix (the former with the better planar stage):
//   N = 1  never: KC = 4368: 18.4 / 20.9, KC = 37440: 122 / 139
//   N = 2  KC = 2160: 20.3 / 23.6  KC = 3168: 27.7 / 26.9  KC = 4368: 32.7 / 28.5
//   N = 3  KC = 720: 18.1 / 21.8   KC = 1344: 22.8 / 22.3  KC = 13248: 207 / 105
//   N = 4  KC = 720: 29.9 / 31.1   KC = 1344: 50.3 / 31.8  KC = 3168: 117 / 46
//   N = 5  KC = 288: 34.0 / 41.4   KC = 720: 50.9 / 42.0   KC = 2160: 134 / 55
inline bool curved_mma_preferred(int N, int KC) {
  constexpr int from[6] = {0, 0, 3000, 1100, 1000, 400};
  return N >= 2 && N <= 5 && KC >= from[N];
}
bbw_status curved_mma_prepare(int N, CurvedMma &A);
bbw_status curved_mma_stage(int N, const CurvedMma &A, const float *Qold, float *Qnew, float *res,
                            cudaStream_t st);
// point data and bounds from the compact rows of CurvedStageArgs (device);
// legacy stream, ended on return
bbw_status curved_mma_points(const CurvedStageArgs &S, const CurvedMma &A, float *gq, float *fq,
                             float *jq, float *bound);

}  // namespace bbw
