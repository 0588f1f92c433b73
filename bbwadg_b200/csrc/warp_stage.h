// Host-visible description of a prepared warp-matrix stage launch
// (warp_stage.cuh, kernels_warp.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "bbwadg.h"

namespace bbw {

// What the matrix unit's rounding toward zero takes off a sum of products on
// average, relative to it (half an ulp: 3.65e-8 measured over 10^6 sums of 16).
// Operators are packed larger by this, so contractions are free of a mean error.
constexpr double kRoundingBias = 3.65e-8;
// top byte of FP16 bits, rounded: sign, five bits of exponent, three significant bits
__host__ __device__ inline uint8_t rest_byte(uint16_t bits) { return (uint8_t)((bits + 0x80u) >> 8); }

// which form of the stage a context runs (auto: stage_form's rule)
enum WarpForm { WARP_AUTO = 0, WARP_SINGLE = 1, WARP_GROUP = 2 };
// where the group form's operators are: all in L2, all in shared memory, or the
// rests in shared memory and the words in L2
enum OpsPlace { OPS_L2 = 0, OPS_SHARED = 1, OPS_RESTS = 2 };

struct WarpPlan {
  bool single = false, group = false;  // forms this context's sizes allow
  int pinned = WARP_AUTO;              // form chosen by the autotuner or the caller
  bool warp_ops = false;               // operators staged in shared memory
  int group_ops = OPS_L2;
  int products = 4;      // 4: FP32 contexts (with the rest), 3: split FP16
  int N = 0, K = 0, K0 = 0, Kc = 0, Nq = 0, bc = 0, S = 1, nsm = 148, max_ctas = 0;
  bool chained = false;  // launched right behind another stage kernel
  int pat_off = 0, table_ints = 0;
  int oDt = 0, oL = 0, oLt = 0, oV = 0, oVt = 0, oP = 0, oM = 0, ops_n = 0;
  float iD = 1.f, iL = 1.f, iV = 1.f, iP = 1.f, vnorm = 1.f;
  const float *geo = nullptr, *c2p = nullptr, *c2max = nullptr;
  const int *nbr = nullptr, *tables = nullptr;
  const uint4 *ops = nullptr;
  const int *src_tile = nullptr, *src_elem = nullptr;
  const float *src_vec = nullptr;
  float f0 = 0.f, tR = 0.f, samp = 0.f;
  const double *time = nullptr;
};

// Operators as FP16 pairs and a rest in the fragment order of the stage's B
// operands.
// Indices run in blocks of eight; a pair of blocks (16 nodes) interleaves so
// that one lane holds four consecutive nodes, an odd last block is in order
// (warp_node).  A k16 tile gives lane l (hi, hi, lo, lo) of operator row l/4
// and column pairs 2(l%4) of the pair's two blocks; a k8 tile (hi, lo).  The rests
// follow as a plane of their own in the same order, a byte per entry (at oM;
// four-product plans only).
// Order: D [3][KP][NB] and its k8 tiles [3][NB], LIFT [4][FP][NB] and [4][NB],
// Vq [chunk][KP][2] and [chunk][2], Pq [chunk][NB].  Sets the offsets, inverse
// scales and vnorm of the plan.
// Device kernels pack them.
//
// A run of tiles: outer matrices A + o * stride (column-major nr x nc, device), nk
// column pairs (k16) or the odd last block (k8) from k0 on, nj row blocks shifted
// by o * row_step, order [outer][k][row block]; nrp, ncp: extents whose blocks the
// indices run over, at: uint4 offset of the first tile, s: scale.
struct PackRegion {
  const float *A;
  size_t stride;
  int nr, nc, nrp, ncp, outer, nk, nj, k0, row_step, at;
  bool k16;
  float s;
  __host__ __device__ int tiles() const { return outer * nk * nj; }
  int end() const { return at + tiles() * (k16 ? 32 : 16); }
};
// common power-of-two scale of n operators of `len` values (host)
float split_scale(const float *const *A, int n, size_t len);
// Tiles of one column-major nr x nc operator, appended to out: split_rows
// with its rows in chunks of 16 ([chunk][k16 step][2], then the k8 tails [chunk][2]),
// split_columns with its columns in chunks of 16 ([chunk][row block]).
void split_rows(std::vector<PackRegion> &out, const float *A, int nr, int nc, float s, int &off,
                int &off_tail);
void split_columns(std::vector<PackRegion> &out, const float *A, int nr, int nc, float s, int &off);
// words to ops and rests to rests (null: none)
bbw_status pack_operators(const std::vector<PackRegion> &regions, uint4 *ops, uint4 *rests);
// *ops is the context's to free, also on failure
bbw_status warp_pack(WarpPlan &pl, const std::vector<float> *D, const std::vector<float> &LIFT,
                     const std::vector<float> &Vq, const std::vector<float> &Pq, uint4 **ops);
// Sets the forms that fit (pl.single, pl.group).
bbw_status warp_prepare(WarpPlan &pl);
// The form for `elements` (elements of this context times shots) when none is
// pinned; WARP_AUTO: the CTA-wide stages.  One warp and group give the same
// results bit for bit, the CTA-wide stages the same to FP32 rounding: whether the
// arithmetic is the matrix units' depends on N and `whole` only, the elements of
// the whole mesh times shots, of which the context may be a part
// (bbw_set_whole_mesh), so the parts of a cut mesh give the uncut one's bits.  It
// does not depend on the grid limit either.  us per stage, CTA-wide FP32 / one
// warp / group:
//   N = 1  K = 6000: 8.2 / 6.5 / -      K = 93750: 57 / 29 / -
//   N = 2  K = 1296: 5.7 / 9.4 / -      K = 6000: 11.9 / 9.5 / -
//   N = 3  K = 3072: 9.4 / 11.2 / -     K = 6000: 17.6 / 11.1 / -
//   N = 4  K = 6: 15.6 / - / 9.9        K = 3072: 16.8 / 18.2 / 12.7  K = 10368: 43.8 / 22.6 / 34
//   N = 5  K = 6: 21.0 / - / 10.3       K = 3072: 23.8 / - / 14.4     K = 196608: 878 / - / 432
//   N = 6  K = 6: 73 / - / 17.7         K = 24576: 475 / - / 125
//   N = 7  K = 6: 112 / - / 19.3        K = 24576: 736 / - / 212
// and with the package's own rules N = 5, 216 points K = 6: 53.9 / - / 15.2, K = 24576:
// 335 / - / 96; N = 6, 343 points, K = 10368: 289 / - / 72 (before the rests).
// One warp per tile pays once there are about two tiles per SM; the group
// form, three tiles or more per SM at a time, up to the tiles of its first wave
// at N = 4 (four per SM), and at every size above.
inline int stage_form(const WarpPlan &pl, long long elements, long long whole) {
  if (pl.pinned != WARP_AUTO) return pl.pinned;
  if (pl.group && (pl.N >= 5 || elements / 16 <= 4LL * pl.nsm)) return WARP_GROUP;
  return pl.single && (pl.N >= 4 || whole / 16 > 2LL * pl.nsm) ? WARP_SINGLE : WARP_AUTO;
}
bbw_status warp_launch(const WarpPlan &pl, int form, const float *Qin, float *Qout, float *res,
                       float fa, float fb, float fdt, float cstage, cudaStream_t st);
// geometry records [K + 16][28] of the tensor-core and warp-matrix stages (device
// pointers): fgeo 16 | vgeo 9 | pad, a tile's worth of zero records at the end
// The setup kernels (pack_operators, geometry_records, warp_medium) run on the
// legacy stream, behind the copies and fills that made their arguments; the
// contexts' streams do not wait for that stream, so setup_done comes before
// the first launch on them.
bbw_status setup_done(const char *what);
bbw_status geometry_records(int K, const float *vgeo, const float *fgeo, float *geo);
// c2max[k] = max_q |c2q[k][q]|; c2p[k]: c2q[k] padded with zeros to a multiple of 16
bbw_status warp_medium(int K, int Nq, const float *c2q, float *c2max, float *c2p);

}  // namespace bbw
