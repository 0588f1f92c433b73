// Host side of the warp-matrix stage (warp_stage.cuh): operator packing,
// dispatch over N, per-element medium bounds.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "warp_mma.cuh"

namespace bbw {

#define BBW_DECL(form, n)                                                                       \
  bbw_status form##_launch_##n(const WarpPlan &, const float *, float *, float *, float, float, \
                               float, float, cudaStream_t);                                     \
  bbw_status form##_prepare_##n(WarpPlan &);
BBW_DECL(warp, 1) BBW_DECL(warp, 2) BBW_DECL(warp, 3) BBW_DECL(warp, 4)
BBW_DECL(group, 4) BBW_DECL(group, 5) BBW_DECL(group, 6) BBW_DECL(group, 7)
#undef BBW_DECL

bbw_status warp_launch(const WarpPlan &pl, int form, const float *Qin, float *Qout, float *res,
                       float fa, float fb, float fdt, float cstage, cudaStream_t st) {
  switch (pl.N + 16 * form) {
#define CASE(f, form, n) \
  case n + 16 * f: return form##_launch_##n(pl, Qin, Qout, res, fa, fb, fdt, cstage, st);
    CASE(WARP_SINGLE, warp, 1)
    CASE(WARP_SINGLE, warp, 2)
    CASE(WARP_SINGLE, warp, 3)
    CASE(WARP_SINGLE, warp, 4)
    CASE(WARP_GROUP, group, 4)
    CASE(WARP_GROUP, group, 5)
    CASE(WARP_GROUP, group, 6)
    CASE(WARP_GROUP, group, 7)
#undef CASE
  }
  return set_error(BBW_ERR_UNSUPPORTED, "warp-matrix stage: N out of range");
}

bbw_status warp_prepare(WarpPlan &pl) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  pl.nsm = nsm > 0 ? nsm : 148;
  bbw_status a = BBW_ERR_UNSUPPORTED, b = BBW_ERR_UNSUPPORTED;
  switch (pl.N) {
    case 1: a = warp_prepare_1(pl); break;
    case 2: a = warp_prepare_2(pl); break;
    case 3: a = warp_prepare_3(pl); break;
    case 4: a = warp_prepare_4(pl), b = group_prepare_4(pl); break;
    case 5: b = group_prepare_5(pl); break;
    case 6: b = group_prepare_6(pl); break;
    case 7: b = group_prepare_7(pl); break;
  }
  if (a != BBW_OK && a != BBW_ERR_UNSUPPORTED) return a;
  if (b != BBW_OK && b != BBW_ERR_UNSUPPORTED) return b;
  pl.single = a == BBW_OK, pl.group = b == BBW_OK;
  return BBW_OK;
}

// power of two that brings the largest |a| into [2^14, 2^15): the rest of a pair,
// 2^-24 of it, then is a byte of three significant bits
static float operator_scale(const float *a, size_t n) {
  float m = 0.f;
  for (size_t i = 0; i < n; ++i) m = std::max(m, std::fabs(a[i]));
  if (!(m > 0.f) || !std::isfinite(m)) return 1.f;
  int e = 0;
  std::frexp(m, &e);  // m in [2^(e-1), 2^e)
  return std::ldexp(1.f, std::min(std::max(15 - e, -100), 100));
}

// one thread per lane of a tile of the region r
template <bool K16>
__global__ void k_pack(const PackRegion r, uint4 *ops, uint4 *rests) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, tile = i >> 5, lane = i & 31;
  if (tile >= r.tiles()) return;
  const int j = tile % r.nj, k = tile / r.nj % r.nk, o = tile / (r.nj * r.nk);
  const float *A = r.A + (size_t)o * r.stride;
  const int row = slot_index(r.nrp, j + o * r.row_step, lane >> 2);
  uint32_t *w = reinterpret_cast<uint32_t *>(ops + r.at);
  uint32_t *m = rests ? reinterpret_cast<uint32_t *>(rests) + r.at : nullptr;
  split_tile<K16>(w, m, i, r.k0 + k, 2 * (lane & 3), r.s, [&](int b, int slot) {
    const int col = slot_index(r.ncp, b, slot);
    return row < r.nr && col < r.nc ? __ldg(A + row + (size_t)col * r.nr) : 0.f;
  });
}

bbw_status pack_operators(const std::vector<PackRegion> &regions, uint4 *ops, uint4 *rests) {
  for (const PackRegion &r : regions) {
    const int n = r.tiles() * 32;
    if (n == 0) continue;
    if (r.k16) k_pack<true><<<(n + 127) / 128, 128>>>(r, ops, rests);
    else k_pack<false><<<(n + 127) / 128, 128>>>(r, ops, rests);
  }
  return check_launch("split operators");
}

float split_scale(const float *const *A, int n, size_t len) {
  float s = operator_scale(A[0], len);
  for (int i = 1; i < n; ++i) s = std::min(s, operator_scale(A[i], len));
  return s;
}

// appends a region behind the ones before it; returns its offset
static int append(std::vector<PackRegion> &out, PackRegion r) {
  r.at = out.empty() ? 0 : out.back().end();
  out.push_back(r);
  return r.at;
}

void split_rows(std::vector<PackRegion> &out, const float *A, int nr, int nc, float s, int &off,
                int &off_tail) {
  const int nch = (nr + 15) / 16, NB = (nc + 7) / 8, KP = NB / 2, KT = NB % 2;
  PackRegion r{A, 0, nr, nc, 16 * nch, nc, nch, KP, 2, 0, 2, 0, true, s};
  off = append(out, r);
  r.k0 = 2 * KP, r.nk = KT, r.k16 = false;
  off_tail = append(out, r);
}

void split_columns(std::vector<PackRegion> &out, const float *A, int nr, int nc, float s, int &off) {
  const int nch = (nc + 15) / 16, NB = (nr + 7) / 8;
  off = append(out, {A, 0, nr, nc, nr, 16 * nch, 1, nch, NB, 0, 0, 0, true, s});
}

// blocks of the columns of n matrices A + i * stride, [i][k][block], then the odd last ones
static void split_blocks(std::vector<PackRegion> &out, const float *A, size_t stride, int n, int nr,
                         int nc, float s, int &off, int &off_tail) {
  const int RB = (nr + 7) / 8, NB = (nc + 7) / 8, KP = NB / 2, KT = NB % 2;
  PackRegion r{A, stride, nr, nc, nr, nc, n, KP, RB, 0, 0, 0, true, s};
  off = append(out, r);
  r.k0 = 2 * KP, r.nk = KT, r.k16 = false;
  off_tail = append(out, r);
}

bbw_status warp_pack(WarpPlan &pl, const std::vector<float> *D, const std::vector<float> &LIFT,
                     const std::vector<float> &Vq, const std::vector<float> &Pq, uint4 **ops) {
  const int N = pl.N, Np = np_of(N), Nfp = nfp_of(N), Nq = pl.Nq;
  const float *Dp[3] = {D[0].data(), D[1].data(), D[2].data()};
  const float sD = split_scale(Dp, 3, D[0].size()), sL = operator_scale(LIFT.data(), LIFT.size());
  const float sV = operator_scale(Vq.data(), Vq.size()), sP = operator_scale(Pq.data(), Pq.size());
  // the operators themselves sit behind the tiles in the same buffer: the device
  // packs them (on eight host threads creation took up to 7 ms longer where other
  // work held these up)
  std::vector<float> all;
  for (const std::vector<float> *v : {&D[0], &D[1], &D[2], &LIFT, &Vq, &Pq}) all.insert(all.end(), v->begin(), v->end());
  auto regions = [&](const float *A) {
    std::vector<PackRegion> r;
    const size_t n = (size_t)Np * Np;
    int none = 0;
    split_blocks(r, A, n, 3, Np, Np, sD, none, pl.oDt);
    split_blocks(r, A + 3 * n, (size_t)Nfp * Np, 4, Np, Nfp, sL, pl.oL, pl.oLt);
    const float *V = A + 3 * n + (size_t)4 * Nfp * Np;
    split_rows(r, V, Nq, Np, sV, pl.oV, pl.oVt);
    split_columns(r, V + (size_t)Nq * Np, Np, Nq, sP, pl.oP);
    return r;
  };
  pl.oM = regions(nullptr).back().end();
  pl.ops_n = pl.oM + (pl.products == 4 ? pl.oM / 4 : 0);
  cudaError_t e = cudaMalloc((void **)ops, (size_t)pl.ops_n * 16 + all.size() * sizeof(float));
  if (e != cudaSuccess) return set_cuda_error(e, "split operators");
  float *dense = reinterpret_cast<float *>(*ops + pl.ops_n);
  e = cudaMemcpy(dense, all.data(), all.size() * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return set_cuda_error(e, "split operators");
  const bbw_status st = pack_operators(regions(dense), *ops, pl.products == 4 ? *ops + pl.oM : nullptr);
  if (st != BBW_OK) return st;
  pl.iD = 1.f / sD, pl.iL = 1.f / sL, pl.iV = 1.f / sV, pl.iP = 1.f / sP;
  double vn = 0.0;
  for (int q = 0; q < Nq; ++q) {
    double s = 0.0;
    for (int n = 0; n < Np; ++n) s += std::fabs((double)Vq[q + (size_t)n * Nq]);
    vn = std::max(vn, s);
  }
  // twice the bound, as for the divergence: rounding cannot reach 2^16
  pl.vnorm = (float)(2.0 * vn);
  return BBW_OK;
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

// one thread per float of the records: fgeo 16 | vgeo 9 | pad 3, rows past K zero
__global__ void k_records(int K, const float *__restrict__ vgeo, const float *__restrict__ fgeo,
                          float *__restrict__ geo) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long k = i / 28;
  const int c = (int)(i - k * 28);
  if (k >= K + 16) return;
  geo[i] = k >= K || c >= 25 ? 0.f : c < 16 ? fgeo[k * 16 + c] : vgeo[k * 9 + c - 16];
}

bbw_status setup_done(const char *what) {
  return set_cuda_error(cudaStreamSynchronize(nullptr), what);
}

bbw_status geometry_records(int K, const float *vgeo, const float *fgeo, float *geo) {
  const long long n = (long long)(K + 16) * 28;
  k_records<<<(int)((n + 255) / 256), 256>>>(K, vgeo, fgeo, geo);
  return check_launch("geometry records");
}

bbw_status warp_medium(int K, int Nq, const float *c2q, float *c2max, float *c2p) {
  k_medium<<<(K + 7) / 8, 256>>>(K, Nq, (Nq + 15) / 16 * 16, c2q, c2max, c2p);
  return check_launch("medium bound");
}

}  // namespace bbw
