// Host side of the warp-matrix stage (warp_stage.cuh): operator packing,
// dispatch over N, per-element medium bounds.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "device_common.cuh"
#include "internal.h"
#include "warp_stage.h"

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

// operator entry times its scale (1 + kRoundingBias) as FP16 hi and lo and the
// top byte of an FP16 rest
struct Parts {
  std::vector<uint32_t> w;  // hi | lo << 16
  std::vector<uint8_t> m;
  int nr = 0;
};
static void split_entry(double a, uint32_t &w, uint8_t &m) {
  const __half h = __double2half(a), l = __double2half(a - __half2float(h));
  w = (uint32_t)__half_as_ushort(h) | (uint32_t)__half_as_ushort(l) << 16;
  m = rest_byte(__half_as_ushort(__double2half(a - __half2float(h) - __half2float(l))));
}
// the column-major nr x nc matrix A times s
static void split_matrix(Parts &p, const float *A, int nr, int nc, float s) {
  const size_t n = (size_t)nr * nc;
  p.nr = nr, p.w.resize(n), p.m.resize(n);
  for (size_t i = 0; i < n; ++i) split_entry((double)A[i] * s * (1.0 + kRoundingBias), p.w[i], p.m[i]);
}

// index of slot c of block b when n indices are stored in blocks of eight
static int warp_node(int n, int b, int c) {
  const int nb = (n + 7) / 8;
  if (b == nb - 1 && nb % 2) return 8 * b + c;
  return 16 * (b / 2) + 4 * (c / 2) + 2 * (b % 2) + c % 2;
}

// tile of row block j and columns of pair (k16) or block (k8) k of the matrix
// at p.w + at (nr x nc), zero outside; nrp, ncp: extents whose blocks the
// indices run over
struct PackTile {
  const Parts *p;
  size_t at;
  int nr, nc, nrp, ncp, j, k;
  bool k16;
};

static void pack_tile(const PackTile &q, uint32_t *out, uint8_t *rest) {
  for (int lane = 0; lane < 32; ++lane) {
    const int r = warp_node(q.nrp, q.j, lane / 4), c = 2 * (lane % 4);
    // entries c and c + 1 of block b: words of hi, lo; bytes of the rest
    auto words = [&](int b, uint32_t &hi, uint32_t &lo, uint8_t *m) {
      uint32_t x[2];
      for (int i = 0; i < 2; ++i) {
        const int col = warp_node(q.ncp, b, c + i);
        const bool in = r < q.nr && col < q.nc;
        const size_t e = q.at + r + (size_t)col * q.nr;
        x[i] = in ? q.p->w[e] : 0u, m[i] = in ? q.p->m[e] : 0;
      }
      hi = (x[0] & 0xffffu) | x[1] << 16, lo = x[0] >> 16 | (x[1] & 0xffff0000u);
    };
    if (q.k16) {
      uint32_t *o = out + 4 * lane;
      words(2 * q.k, o[0], o[2], rest + 4 * lane);
      words(2 * q.k + 1, o[1], o[3], rest + 4 * lane + 2);
    } else {
      words(q.k, out[2 * lane], out[2 * lane + 1], rest + 2 * lane);
    }
  }
}

float split_scale(const float *const *A, int n, size_t len) {
  float s = operator_scale(A[0], len);
  for (int i = 1; i < n; ++i) s = std::min(s, operator_scale(A[i], len));
  return s;
}

static void append(SplitOps &out, const PackTile &q) {
  const size_t n = q.k16 ? 128 : 64, at = out.w.size();
  out.w.resize(at + n), out.m.resize(at + n);
  pack_tile(q, &out.w[at], &out.m[at]);
}

void split_rows(SplitOps &out, const float *A, int nr, int nc, float s, int &off, int &off_tail) {
  const int nch = (nr + 15) / 16, NB = (nc + 7) / 8, KP = NB / 2, KT = NB % 2;
  Parts p;
  split_matrix(p, A, nr, nc, s);
  off = (int)(out.w.size() / 4);
  for (int c = 0; c < nch; ++c)
    for (int k = 0; k < KP; ++k)
      for (int h = 0; h < 2; ++h) append(out, {&p, 0, nr, nc, 16 * nch, nc, 2 * c + h, k, true});
  off_tail = (int)(out.w.size() / 4);
  for (int c = 0; c < nch && KT; ++c)
    for (int h = 0; h < 2; ++h) append(out, {&p, 0, nr, nc, 16 * nch, nc, 2 * c + h, 2 * KP, false});
}

void split_columns(SplitOps &out, const float *A, int nr, int nc, float s, int &off) {
  const int nch = (nc + 15) / 16, NB = (nr + 7) / 8;
  Parts p;
  split_matrix(p, A, nr, nc, s);
  off = (int)(out.w.size() / 4);
  for (int c = 0; c < nch; ++c)
    for (int j = 0; j < NB; ++j) append(out, {&p, 0, nr, nc, nr, 16 * nch, j, c, true});
}

std::vector<uint32_t> SplitOps::words() const {
  std::vector<uint32_t> all(w);
  all.resize(w.size() + m.size() / 4);
  std::memcpy(all.data() + w.size(), m.data(), m.size());
  return all;
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
  Parts D3[3], L, V, P;
#pragma omp parallel for schedule(dynamic) num_threads(6) if (Np > 30)
  for (int i = 0; i < 6; ++i) {
    if (i < 3) split_matrix(D3[i], D[i].data(), Np, Np, sD);
    else if (i == 3) split_matrix(L, LIFT.data(), Np, 4 * Nfp, sL);
    else if (i == 4) split_matrix(V, Vq.data(), Nq, Np, sV);
    else split_matrix(P, Pq.data(), Np, Nq, sP);
  }
  std::vector<PackTile> tiles;
  std::vector<size_t> offset;
  size_t words = 0;
  auto add = [&](const PackTile &q) {
    tiles.push_back(q), offset.push_back(words);
    words += q.k16 ? 128 : 64;
  };
  auto at = [&]() { return (int)(words / 4); };
  for (int d = 0; d < 3; ++d)
    for (int k = 0; k < KP; ++k)
      for (int j = 0; j < NB; ++j) add({&D3[d], 0, Np, Np, Np, Np, j, k, true});
  pl.oDt = at();
  for (int d = 0; d < 3 && KT; ++d)
    for (int j = 0; j < NB; ++j) add({&D3[d], 0, Np, Np, Np, Np, j, 2 * KP, false});
  pl.oL = at();
  auto face = [&](int f) { return (size_t)f * Nfp * Np; };
  for (int f = 0; f < 4; ++f)
    for (int k = 0; k < FP; ++k)
      for (int j = 0; j < NB; ++j) add({&L, face(f), Np, Nfp, Np, Nfp, j, k, true});
  pl.oLt = at();
  for (int f = 0; f < 4 && FT; ++f)
    for (int j = 0; j < NB; ++j) add({&L, face(f), Np, Nfp, Np, Nfp, j, 2 * FP, false});
  pl.oV = at();
  for (int c = 0; c < nch; ++c)
    for (int k = 0; k < KP; ++k)
      for (int h = 0; h < 2; ++h) add({&V, 0, Nq, Np, Nq16, Np, 2 * c + h, k, true});
  pl.oVt = at();
  for (int c = 0; c < nch && KT; ++c)
    for (int h = 0; h < 2; ++h) add({&V, 0, Nq, Np, Nq16, Np, 2 * c + h, 2 * KP, false});
  pl.oP = at();
  for (int c = 0; c < nch; ++c)
    for (int j = 0; j < NB; ++j) add({&P, 0, Np, Nq, Np, Nq16, j, c, true});
  pl.oM = at();
  SplitOps all;
  all.w.resize(words), all.m.resize(words);
  const long long nt = (long long)tiles.size();
#pragma omp parallel for schedule(static) num_threads(8) if (nt > 128)
  for (long long i = 0; i < nt; ++i) pack_tile(tiles[i], &all.w[offset[i]], &all.m[offset[i]]);
  out = pl.products == 4 ? all.words() : std::move(all.w);
  pl.ops_n = (int)(out.size() / 4);
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

// one thread per float of the records: fgeo 16 | vgeo 9 | pad 3, rows past K zero
__global__ void k_records(int K, const float *__restrict__ vgeo, const float *__restrict__ fgeo,
                          float *__restrict__ geo) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long k = i / 28;
  const int c = (int)(i - k * 28);
  if (k >= K + 16) return;
  geo[i] = k >= K || c >= 25 ? 0.f : c < 16 ? fgeo[k * 16 + c] : vgeo[k * 9 + c - 16];
}

bbw_status geometry_records(int K, const float *vgeo, const float *fgeo, float *geo) {
  const long long n = (long long)(K + 16) * 28;
  k_records<<<(int)((n + 255) / 256), 256>>>(K, vgeo, fgeo, geo);
  const bbw_status s = check_launch("geometry records");
  return s != BBW_OK ? s : set_cuda_error(cudaStreamSynchronize(nullptr), "geometry records");
}

bbw_status warp_medium(int K, int Nq, const float *c2q, float *c2max, float *c2p) {
  k_medium<<<(K + 7) / 8, 256>>>(K, Nq, (Nq + 15) / 16 * 16, c2q, c2max, c2p);
  const bbw_status s = check_launch("medium bound");
  return s != BBW_OK ? s : set_cuda_error(cudaStreamSynchronize(nullptr), "medium bound");
}

}  // namespace bbw
