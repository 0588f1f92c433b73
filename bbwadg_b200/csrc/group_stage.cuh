// One LSRK stage with every contraction on warp-level matrix instructions
// (warp_mma.cuh), a group of three to eight warps per 16-element tile.
//
// Replaces rk_volume + rk_surface + rk_update_WADG of the reference
// (cpp/okl/WaveKernels.okl:44-260, cpp/okl/WaveKernelsWADG.okl:1760-1887).
//
// The group's warps split the operator rows and hand the next contraction's
// operand to each other as ready fragments in shared memory, with a named
// barrier between phases.  Against one warp per tile (warp_stage.cuh) a tile's
// chain is three to eight times shorter, which counts where a mesh has few tiles
// or an element much work.  The results are the same bit for bit.  us per
// stage, CTA-wide FP32 stage / group: N = 5, K = 3072: 23.8 / 14.4, K = 196608: 878 /
// 432; N = 6, K = 24576: 475 / 125; N = 7: 736 / 212; N = 4, K = 3072: 16.8 / 12.7 (one
// warp per tile 18.2).  Bound by instruction and L1 wavefront rate together
// (issue 36 %, L1 data pipe 57 %, tensor 28 %; before the rests, without the products
// 261 of 411 us, without global loads 399, without stores 325, N = 5, K = 196608).
#pragma once
#include <vector>

#include "warp_mma.cuh"

namespace bbw {

template <int N>
struct GroupCfg {
  static constexpr int Np = NP(N), Nfp = NFP(N), EW = 4 * Np;
  // blocks of eight nodes: pairs of them are the k16 steps, an odd last one
  // is a k8 step (same for the face nodes)
  static constexpr int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2;
  static constexpr int FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  // a unit of work is a pair of blocks (or the odd last one): one for each of the
  // group's GW warps, whose old state stays in registers; NG groups per CTA.  us per
  // stage at K = 24576 with three or four warps and two units each, 168 registers /
  // one unit per warp: N = 6 145 / 123, N = 7 254 / 178 (one group of 255 registers;
  // two of 128: 205).
  static constexpr int U = KP + KT;
  static constexpr int GW = U;  // 3, 4, 6, 8 at N = 4 .. 7
  static constexpr int NG = N <= 6 ? 12 / GW : 1;
  static constexpr int W = GW * NG, T = 32 * W;
  // operators in shared memory when they fit; else their rests (a fifth of them;
  // rests from L2 as well / from shared memory: N = 7, K = 24576 219 / 207 us per stage)
  static constexpr bool OPS = N <= 5;
  static constexpr int V = Np % 4 == 0 ? 4 : Np % 2 == 0 ? 2 : 1;  // vector width of a row
  // state tile of a group: rows of 4 Np floats, padded so that two rows of a
  // pair start 16 banks apart (a 16-byte access serves two rows at a time).
  // Once read, it holds the split p and contravariant velocities.
  static constexpr int ODD = V == 4 ? (48 - EW % 32) % 32 : 0;
  static constexpr int ROWS = 16 * EW + 8 * ODD;
  static constexpr int TILE = ROWS > 512 * NB ? ROWS : 512 * NB;
  __host__ __device__ static constexpr int row(int e) { return e * EW + ((e + 1) >> 1) * ODD; }
  // split face fluxes, then split rhs_p over them
  static constexpr int FLUX = 4 * FB * 128;
  static_assert(NB <= 4 * FB, "rhs_p fits over the fluxes");
  static constexpr int RC = GW == 6 ? 12 : 8;  // cubature chunks per round
  static constexpr bool EARLY = !OPS;    // residual of p loaded before the projection
  // a sum's first step sets it instead of adding to zero: fewer instructions, but by
  // the registers it pays at N = 6 only (us per stage added / set: N = 5, K = 196608 432 /
  // 437, N = 6, K = 24576 132 / 125, N = 7 212 / 215)
  static constexpr bool SET = N == 6;
  static constexpr int SCR1 = 8 * FB * 8;      // one warp's face fluxes of eight elements
  static constexpr int WF = RC * 256 > GW * SCR1 ? RC * 256 : GW * SCR1;  // split cubature values
  static constexpr int GEO = 16 * 28;
  static constexpr int MISC = GW * 16 * 4 + GW * 16 + 64;  // maxima of the state, of rhs_p, face scales
  static constexpr int SCR = TILE + FLUX + WF + GEO + MISC;  // floats per group
};

// Gather of face f of eight elements h8 .. h8 + 7 of the tile, nodes I0 .. I0 +
// NI - 1: EPI elements per pass, lane = (element, node), so a pass reads the
// face nodes of a neighbour's row together.
template <int N, int I0, int NI, bool CHAINED>
struct TileFace {
  using C = GroupCfg<N>;
  static constexpr int EPI = NI >= 32 ? 1 : (32 / NI > 8 ? 8 : 32 / NI);
  static constexpr int IT = (8 + EPI - 1) / EPI;
  float X[IT][4];
  uint32_t walls;

  __device__ __forceinline__ static int sub(int lane) { return lane / NI < EPI ? lane / NI : 0; }
  __device__ __forceinline__ static int node(int lane) {
    return lane / NI < EPI ? I0 + lane % NI : I0;
  }
  __device__ __forceinline__ static int elem(int it, int lane) {
    const int e = it * EPI + sub(lane);
    return IT * EPI > 8 && it == IT - 1 ? min(e, 7) : e;
  }

  // code: neighbour codes of the half's faces, one per lane (element * 4 + face)
  __device__ __forceinline__ void load(const float *__restrict__ Qs, const int *sTab, int pat_off,
                                       int f, int code, int lane) {
    const int i = node(lane);
    walls = 0;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int cd = __shfl_sync(0xffffffffu, code, elem(it, lane) * 4 + f);
      const int pat = cd & 255;
      const bool wall = pat == 255;
      walls |= wall ? 1u << it : 0u;
      // a wall's + trace is the own face node (the table starts with Fmask)
      const int nn = sTab[(wall ? f * C::Nfp : pat_off + pat * C::Nfp) + i];
      const float *x = Qs + (size_t)(cd >> 8) * C::EW + nn;
#pragma unroll
      for (int c = 0; c < 4; ++c) X[it][c] = load_trace<CHAINED>(x + c * C::Np);
    }
  }
  // upwind pressure flux to sF[element][8 FB].  A wall's + trace is the own
  // one with the pressure (p = 0 wall) or the velocity (rigid) reversed.
  __device__ __forceinline__ void flux(int bc, const float *sQ, const float *sGeo, const int *sFm,
                                       float *sF, int f, int h8, int lane) const {
    const bool act = lane / NI < EPI;
    const int i = node(lane), own = sFm[f * C::Nfp + i];
    const float wp = bc == BBW_BC_PRESSURE_RELEASE ? -1.f : 1.f, wu = -wp;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = elem(it, lane);
      const float *m = sQ + C::row(h8 + e) + own;
      const float4 g = *reinterpret_cast<const float4 *>(sGeo + (h8 + e) * 28 + 4 * f);
      const bool wall = walls >> it & 1u;
      const float sp = wall ? wp : 1.f, su = wall ? wu : 1.f;
      const float dp = fmaf(sp, X[it][0], -m[0]);
      float un = fmaf(su, X[it][1], -m[C::Np]) * g.y;
      un = fmaf(fmaf(su, X[it][2], -m[2 * C::Np]), g.z, un);
      un = fmaf(fmaf(su, X[it][3], -m[3 * C::Np]), g.w, un);
      const float fl = .5f * g.x * (dp - un);
      if (IT * EPI > 8 && it == IT - 1) {
        if (act && it * EPI + sub(lane) < 8) sF[e * (8 * C::FB) + i] = fl;
      } else {
        if (act) sF[e * (8 * C::FB) + i] = fl;
      }
    }
  }
};

template <int N, bool CHAINED, bool WIDE>
struct TileHalf;
template <int N, bool CHAINED>
struct TileHalf<N, CHAINED, false> {
  TileFace<N, 0, NFP(N), CHAINED> a;
  template <class... A>
  __device__ __forceinline__ void load(A... x) { a.load(x...); }
  template <class... A>
  __device__ __forceinline__ void flux(A... x) const { a.flux(x...); }
};
template <int N, bool CHAINED>
struct TileHalf<N, CHAINED, true> {  // more than 32 nodes per face
  TileFace<N, 0, 32, CHAINED> a;
  TileFace<N, 32, (NFP(N) > 32 ? NFP(N) - 32 : 1), CHAINED> b;
  template <class... A>
  __device__ __forceinline__ void load(A... x) { a.load(x...), b.load(x...); }
  template <class... A>
  __device__ __forceinline__ void flux(A... x) const { a.flux(x...), b.flux(x...); }
};

// the eight (pair: M = 2 blocks) or four (M = 1) values of a unit in one field
// for rows a and b, as they sit in memory
template <int M>
struct Unit;
template <>
struct Unit<2> {
  using T = float4;
  __device__ __forceinline__ static int node(int u, int t) { return 16 * u + 4 * t; }
  template <int Np, int V>
  __device__ __forceinline__ static T load(const float *x, int n) { return load4<Np, V>(x, n); }
  template <int Np, int V>
  __device__ __forceinline__ static void store(float *x, int n, const T v) { store4<Np, V>(x, n, v); }
  __device__ __forceinline__ static float max(float m, const T v) { return max4(m, v); }
  // row a (h = 0) or b (h = 1) of the blocks' accumulators
  __device__ __forceinline__ static T row(const float (&c)[2][4], int h) {
    return make_float4(c[0][2 * h], c[0][2 * h + 1], c[1][2 * h], c[1][2 * h + 1]);
  }
  __device__ __forceinline__ static void lsrk(const T r0, const T x, const T q0, const WarpParams &P,
                                              T &r, T &q) {
    lsrk4(r0, x, q0, P, r, q);
  }
  __device__ __forceinline__ static T mix(const T a, const T b, const T c, float x, float y, float z) {
    return make_float4(a.x * x + b.x * y + c.x * z, a.y * x + b.y * y + c.y * z,
                       a.z * x + b.z * y + c.z * z, a.w * x + b.w * y + c.w * z);
  }
  __device__ __forceinline__ static void split(uint4 *a, int u, int lane, const T x, const T y,
                                               float ca, float cb) {
    Frag f;
    split_frag(f, x, y, ca, cb);
    put_frag(a, u, lane, f);
  }
};
template <>
struct Unit<1> {
  using T = float2;
  __device__ __forceinline__ static int node(int u, int t) { return 16 * u + 2 * t; }
  template <int Np, int V>
  __device__ __forceinline__ static T load(const float *x, int n) { return load2<Np, V>(x, n); }
  template <int Np, int V>
  __device__ __forceinline__ static void store(float *x, int n, const T v) { store2<Np, V>(x, n, v); }
  __device__ __forceinline__ static float max(float m, const T v) { return max2(m, v); }
  __device__ __forceinline__ static T row(const float (&c)[1][4], int h) {
    return make_float2(c[0][2 * h], c[0][2 * h + 1]);
  }
  __device__ __forceinline__ static void lsrk(const T r0, const T x, const T q0, const WarpParams &P,
                                              T &r, T &q) {
    r = lsrk2(r0, x, both(P.fa), both(P.fdt));
    q = __ffma2_rn(both(P.fb), r, q0);
  }
  __device__ __forceinline__ static T mix(const T a, const T b, const T c, float x, float y, float z) {
    return make_float2(a.x * x + b.x * y + c.x * z, a.y * x + b.y * y + c.y * z);
  }
  __device__ __forceinline__ static void split(uint4 *a, int u, int lane, const T x, const T y,
                                               float ca, float cb) {
    Frag8 f;
    split_frag(f, x, y, ca, cb);
    put_frag8(a, u, lane, f);
  }
};

template <int N, int PR, int PLACE>
__global__ void __launch_bounds__(GroupCfg<N>::T, 1) k_group_stage(const WarpParams P) {
  using C = GroupCfg<N>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW;
  constexpr int FB = C::FB, FP = C::FP, FT = C::FT, V = C::V, GW = C::GW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = warp / GW, w = warp - grp * GW;
  const int g = lane >> 2, t = lane & 3;
  uint4 *sOps = reinterpret_cast<uint4 *>(smem_raw);
  constexpr bool OPS = PLACE == OPS_SHARED;
  const int nops = OPS ? P.ops_n : PLACE == OPS_RESTS ? P.ops_n - P.oM : 0;
  int *sTab = reinterpret_cast<int *>(sOps + nops);
  float *scr = reinterpret_cast<float *>(sTab + P.table_ints) + grp * C::SCR;
  // operators and tables, all copies in flight with the first tile's
  if constexpr (OPS) stage_async<C::T>(sOps, P.ops, P.ops_n);
  if constexpr (PLACE == OPS_RESTS) stage_async<C::T>(sOps, P.ops + P.oM, nops);
  stage_async<C::T>(reinterpret_cast<uint4 *>(sTab), reinterpret_cast<const uint4 *>(P.tables),
                    P.table_ints / 4);
  float *sQ = scr;                                            // state rows, then
  uint4 *sA = reinterpret_cast<uint4 *>(scr);                 // split p, Ur, Us, Ut
  constexpr int AS = KP * 64 + KT * 32, FS = FP * 64 + FT * 32;  // uint4 per operand, per face
  uint4 *sFr = reinterpret_cast<uint4 *>(scr + C::TILE);      // split face fluxes
  uint4 *sR = sFr;                                            // split rhs_p, once these are consumed
  uint4 *sW = reinterpret_cast<uint4 *>(scr + C::TILE + C::FLUX);    // split c2 Vq rhs_p
  float *sF = scr + C::TILE + C::FLUX + w * C::SCR1;  // before that, face fluxes
  float *sGeo = scr + C::TILE + C::FLUX + C::WF;
  float4 *sMax = reinterpret_cast<float4 *>(sGeo + C::GEO);   // [GW][16] |p|, |u|, |v|, |w|
  float *sMaxR = sGeo + C::GEO + GW * 64, *sInv = sMaxR + GW * 16;  // [GW][16], [4][16]
  const uint4 *ops = OPS ? sOps : P.ops;
  constexpr int PD = PR == 4 ? 5 : PR;  // derivatives: large terms cancel
  constexpr bool SET = C::SET;
  using O16 = Ops<uint4, PR, !OPS, PLACE == OPS_L2>;
  using O8 = Ops<uint2, PR, !OPS, PLACE == OPS_L2>;
  const void *rests = PLACE == OPS_RESTS ? sOps : ops + P.oM;
  const O16 oD(ops, rests, 0, lane), oL(ops, rests, P.oL, lane), oV(ops, rests, P.oV, lane),
      oP(ops, rests, P.oP, lane);
  const O8 oDt(ops, rests, P.oDt, lane), oLt(ops, rests, P.oLt, lane), oVt(ops, rests, P.oVt, lane);
  const int klast = P.Kc - 1;
  const size_t shot_stride = (size_t)P.K * EW;
  const int step = gridDim.x * C::NG;

  // state rows and geometry records of the tile at element kn of shot sh to
  // shared memory, a row per warp
  auto fetch_tile = [&](int sh, int kn) {
    const int ne = min(16, P.Kc - kn);
    const float *src = P.Qin + sh * shot_stride + (size_t)kn * EW;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sQ);
    const uint32_t geo = (uint32_t)__cvta_generic_to_shared(sGeo);
    for (int e = w; e < ne; e += GW)
#pragma unroll
      for (int c = 0; c < Np; c += 32)
        if (c + lane < Np)
          cp_async16(dst + 4 * (C::row(e) + 4 * (c + lane)), src + e * EW + 4 * (c + lane));
    for (int c = w * 32 + lane; c < 16 * 7; c += 32 * GW)
      cp_async16(geo + 16 * c, P.geo + (size_t)kn * 28 + 4 * c);
  };
  auto codes = [&](int kn, int &c0, int &c1) {
    c0 = __ldg(P.nbr + (size_t)min(kn + g, klast) * 4 + t);
    c1 = __ldg(P.nbr + (size_t)min(kn + 8 + g, klast) * 4 + t);
  };

  int it = blockIdx.x * P.bs + grp * P.ws;
  int code0 = 0, code1 = 0;
  int nshot = it / P.ntile, ntl = it - nshot * P.ntile;  // the next item
  if (it < P.nit) codes(P.K0 + ntl * 16, code0, code1);
  // operators from L2 leave nothing to stage early, and the gather's read-only
  // path is worth more (N = 7: 178 against 182 us per stage chained)
  if constexpr (OPS) stage_wait();
  if (it < P.nit) fetch_tile(nshot, P.K0 + ntl * 16);
  cp_async_wait();
  __syncthreads();
  for (; it < P.nit; it += step) {
    const int shot = nshot, k0 = P.K0 + ntl * 16;
    nshot += P.step_shot, ntl += P.step_tile;
    if (ntl >= P.ntile) ntl -= P.ntile, ++nshot;
    const int kn = P.K0 + ntl * 16;  // next item's first element
    const float *Qs = P.Qin + shot * shot_stride;
    const int ka = min(k0 + g, klast), kb = min(k0 + g + 8, klast);
    const bool va = k0 + g < P.Kc, vb = k0 + g + 8 < P.Kc;
    const size_t ea = (size_t)ka * EW, eb = (size_t)kb * EW;
    float *Ra = P.res + shot * shot_stride + ea, *Rb = P.res + shot * shot_stride + eb;
    float *Oa = P.Qout + shot * shot_stride + ea, *Ob = P.Qout + shot * shot_stride + eb;

    if (lane == 0 && w == 0) {  // the next item's inputs on their way to L2
      if (it + step < P.nit) {
        const int ne = min(16, P.Kc - kn);
        const size_t at = nshot * shot_stride + (size_t)kn * EW;
        prefetch_l2(P.Qin + at, (size_t)ne * EW * 4);
        prefetch_l2(P.res + at, (size_t)ne * EW * 4);
        prefetch_l2(P.c2p + (size_t)kn * P.Nq16, (size_t)ne * P.Nq16 * 4);
      }
    }

    // ---- 1. face fluxes, eight elements of one face at a time, and the
    //         maxima of the warp's own nodes
    {
      TileHalf<N, OPS, (Nfp > 32)> x;
      x.load(Qs, sTab, P.pat_off, w >> 1, w & 1 ? code1 : code0, lane);
      cp_async_wait();
      group_sync<GW>(grp);  // the tile has landed
#pragma unroll 1
      for (int r = w; r < 8; r += GW) {
        const int f = r >> 1, h = r & 1;
        if constexpr (FB * 8 > Nfp) {  // columns past Nfp meet zero operator columns
          constexpr int PD = FB * 8 - Nfp;
          for (int i = lane; i < 8 * PD; i += 32) sF[(i / PD) * (8 * FB) + Nfp + i % PD] = 0.f;
        }
        x.flux(P.bc, sQ, sGeo, sTab, sF, f, 8 * h, lane);
        if (r + GW < 8)
          x.load(Qs, sTab, P.pat_off, (r + GW) >> 1, (r + GW) & 1 ? code1 : code0, lane);
        __syncwarp();
        const float *row = sF + g * (8 * FB);
        float4 y[FP > 0 ? FP : 1];
        float2 z = make_float2(0.f, 0.f);
        float m = 0.f;
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          y[k] = *reinterpret_cast<const float4 *>(row + 16 * k + 4 * t);
          m = max4(m, y[k]);
        }
        if constexpr (FT) {
          z = *reinterpret_cast<const float2 *>(row + 16 * FP + 2 * t);
          m = max2(m, z);
        }
        const int sc = scale_field(quad_max(m));
        const float2 cs = both(pow2_field(sc));
        if (t == 0) sInv[f * 16 + 8 * h + g] = pow2_field(254 - sc) * P.iL;
        uint32_t *d = reinterpret_cast<uint32_t *>(sFr + f * FS);
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          uint32_t h0, h1, l0, l1;
          split2(lo2(y[k]), cs, h0, l0);
          split2(hi2(y[k]), cs, h1, l1);
          uint32_t *dk = d + k * 256 + lane * 4 + h;
          dk[0] = h0, dk[2] = h1, dk[128] = l0, dk[130] = l1;
        }
        if constexpr (FT) {
          uint32_t h0, l0;
          split2(z, cs, h0, l0);
          uint32_t *dk = d + FP * 256 + lane * 4 + h;
          dk[0] = h0, dk[2] = l0;
        }
        __syncwarp();
      }
    }
    if (it + step < P.nit) codes(kn, code0, code1);

    const float *Qa = sQ + C::row(ka - k0), *Qb = sQ + C::row(kb - k0);
    // old state of the warp's unit, rows a and b
    float4 qa[4], qb[4];
    {
      float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (KT == 0 || w < KP) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          qa[c] = load4<Np, V>(Qa + c * Np, 16 * w + 4 * t);
          qb[c] = load4<Np, V>(Qb + c * Np, 16 * w + 4 * t);
          m[c] = max4(m[c], qa[c]), m[4 + c] = max4(m[4 + c], qb[c]);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 x = load2<Np, V>(Qa + c * Np, 16 * KP + 2 * t);
          const float2 y = load2<Np, V>(Qb + c * Np, 16 * KP + 2 * t);
          qa[c] = make_float4(x.x, x.y, 0.f, 0.f), qb[c] = make_float4(y.x, y.y, 0.f, 0.f);
          m[c] = max2(m[c], x), m[4 + c] = max2(m[4 + c], y);
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) m[c] = quad_max(m[c]);
      if (t < 2) {
        const float4 v = t == 0 ? make_float4(m[0], m[1], m[2], m[3]) : make_float4(m[4], m[5], m[6], m[7]);
        sMax[w * 16 + g + 8 * t] = v;
      }
    }
    group_sync<GW>(grp);  // fluxes and maxima ready, the rows are read

    // ---- 2. split operands: p and the contravariant velocities
    float pia, pib, uia, uib;  // inverse scales
    {
      float4 ma = sMax[g], mb = sMax[g + 8];
#pragma unroll
      for (int i = 1; i < GW; ++i) {
        const float4 a = sMax[i * 16 + g], b = sMax[i * 16 + g + 8];
        ma = make_float4(fmaxf(ma.x, a.x), fmaxf(ma.y, a.y), fmaxf(ma.z, a.z), fmaxf(ma.w, a.w));
        mb = make_float4(fmaxf(mb.x, b.x), fmaxf(mb.y, b.y), fmaxf(mb.z, b.z), fmaxf(mb.w, b.w));
      }
      const float *A = sGeo + g * 28 + 16, *B = A + 8 * 28;
      const float4 a0 = *reinterpret_cast<const float4 *>(A), a1 = *reinterpret_cast<const float4 *>(A + 4);
      const float4 b0 = *reinterpret_cast<const float4 *>(B), b1 = *reinterpret_cast<const float4 *>(B + 4);
      const float Ga[9] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w, A[8]};
      const float Gb[9] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w, B[8]};
      float Ma = 0.f, Mb = 0.f;  // bounds of the contravariant velocities
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Ma = fmaxf(Ma, fabsf(Ga[3 * c]) * ma.y + fabsf(Ga[3 * c + 1]) * ma.z + fabsf(Ga[3 * c + 2]) * ma.w);
        Mb = fmaxf(Mb, fabsf(Gb[3 * c]) * mb.y + fabsf(Gb[3 * c + 1]) * mb.z + fabsf(Gb[3 * c + 2]) * mb.w);
      }
      // twice the bound: its own rounding cannot bring a value to 2^16
      const int sp = scale_field(ma.x), tp = scale_field(mb.x);
      const int su = scale_field(2.f * Ma), tu = scale_field(2.f * Mb);
      const float cpa = pow2_field(sp), cpb = pow2_field(tp), cua = pow2_field(su), cub = pow2_field(tu);
      pia = -pow2_field(254 - sp) * P.iD, pib = -pow2_field(254 - tp) * P.iD;
      uia = -pow2_field(254 - su) * P.iD, uib = -pow2_field(254 - tu) * P.iD;
      auto split_unit = [&](auto M, int u, const float4 (&xa)[4], const float4 (&xb)[4]) {
        using Un = Unit<decltype(M)::value>;
        if constexpr (decltype(M)::value == 2) {
          Un::split(sA, u, lane, xa[0], xb[0], cpa, cpb);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            Un::split(sA + (c + 1) * AS, u, lane,
                      Un::mix(xa[1], xa[2], xa[3], Ga[3 * c], Ga[3 * c + 1], Ga[3 * c + 2]),
                      Un::mix(xb[1], xb[2], xb[3], Gb[3 * c], Gb[3 * c + 1], Gb[3 * c + 2]), cua, cub);
        } else {
          Un::split(sA, u, lane, lo2(xa[0]), lo2(xb[0]), cpa, cpb);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            Un::split(sA + (c + 1) * AS, u, lane,
                      Un::mix(lo2(xa[1]), lo2(xa[2]), lo2(xa[3]), Ga[3 * c], Ga[3 * c + 1], Ga[3 * c + 2]),
                      Un::mix(lo2(xb[1]), lo2(xb[2]), lo2(xb[3]), Gb[3 * c], Gb[3 * c + 1], Gb[3 * c + 2]),
                      cua, cub);
        }
      };
      if (KT == 0 || w < KP) split_unit(std::integral_constant<int, 2>(), w, qa, qb);
      else split_unit(std::integral_constant<int, 1>(), w, qa, qb);
    }
    group_sync<GW>(grp);  // operands ready

    // ---- 3. gradient, divergence and lift of the warp's unit: update of u, v,
    //         w; rhs_p stays in registers
    float rp[2][4];
    float ma = 0.f, mb = 0.f;  // maxima of rhs_p
    auto rhs_unit = [&](auto M, int u, float (&r)[2][4]) {
      constexpr int m = decltype(M)::value;
      using Un = Unit<m>;
      using T = typename Un::T;
      float rv[3][m][4], rr[m][4], rd[m][4];  // rr: lifted part, rd: divergence
      {
        float d[3][m][4] = {}, dv[m][4] = {};
        // from L2 the next step's operators are loaded during a step's products
        // (48 per warp, about the latency): with the projection's below N = 7
        // 207 -> 183, N = 6 134 -> 129 us per stage
        OpTile<uint4> bk[2][3][m];
        auto load_d = [&](int k) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int i = 0; i < m; ++i)
              bk[k & 1][c][i] = oD[((c * KP + k) * NB + 2 * u + i) * 32];
        };
        if constexpr (!OPS && KP > 0) load_d(0);
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          if (OPS) load_d(k);
          else if (k + 1 < KP) load_d(k + 1);
          const OpTile<uint4> (&b)[3][m] = bk[k & 1];
          const Frag x = get_frag(sA, k, lane);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const Frag y = get_frag(sA + (c + 1) * AS, k, lane);
            mma_pair2<PD, PD>(d[c], x, b[c], dv, y, b[c], SET && k == 0, SET && k == 0 && c == 0);
          }
        }
        if constexpr (KT) {
          OpTile<uint2> b[3][m];
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int i = 0; i < m; ++i) b[c][i] = oDt[(c * NB + 2 * u + i) * 32];
          const Frag8 x = get_frag8(sA, KP, lane);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const Frag8 y = get_frag8(sA + (c + 1) * AS, KP, lane);
            mma_pair2<PD, PD>(d[c], x, b[c], dv, y, b[c]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float *A = sGeo + (g + 8 * h) * 28 + 16;
          const float4 a0 = *reinterpret_cast<const float4 *>(A), a1 = *reinterpret_cast<const float4 *>(A + 4);
          const float s = h ? pib : pia;  // minus the inverse scale
          const float H[9] = {a0.x * s, a0.y * s, a0.z * s, a0.w * s, a1.x * s,
                              a1.y * s, a1.z * s, a1.w * s, A[8] * s};
#pragma unroll
          for (int i = 0; i < m; ++i)
#pragma unroll
            for (int v = 2 * h; v < 2 * h + 2; ++v) {
              const float a = d[0][i][v], b = d[1][i][v], c = d[2][i][v];
#pragma unroll
              for (int x = 0; x < 3; ++x) rv[x][i][v] = H[x] * a + H[3 + x] * b + H[6 + x] * c;
              rd[i][v] = dv[i][v], rr[i][v] = 0.f;
            }
        }
      }
      // residual (and old state) of u, v, w, in flight during the lift
      const int n = Un::node(u, t);
      T ra[3], rb[3], xa[3], xb[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        ra[c] = Un::template load<Np, V>(Ra + (c + 1) * Np, n);
        rb[c] = Un::template load<Np, V>(Rb + (c + 1) * Np, n);
        if constexpr (m == 2) {
          xa[c] = qa[c + 1], xb[c] = qb[c + 1];
        } else {
          xa[c] = lo2(qa[c + 1]), xb[c] = lo2(qb[c + 1]);
        }
      }
      // rolled up but for N = 5 in FP32, by registers; us per stage unrolled / rolled:
      // N = 5 432 / 437 (K = 196608), split FP16 172 / 169 (K = 82944, with the loop over Pq's
      // chunks), N = 4 13.1 / 12.8 (K = 3072), N = 6 137 / 132, N = 7 221 / 212 (K = 24576)
      constexpr int LU = OPS && N == 5 && PR == 4 ? 2 : 1;
#pragma unroll LU
      for (int f0 = 0; f0 < 4; f0 += 2) {
        float L[2][m][4] = {};
        Frag x[2][FP > 0 ? FP : 1];
        OpTile<uint4> b[2][FP > 0 ? FP : 1][m];
        Frag8 x8[2];
        OpTile<uint2> b8[2][m];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int f = f0 + j;
#pragma unroll
          for (int k = 0; k < FP; ++k) {
            x[j][k] = get_frag(sFr + f * FS, k, lane);
#pragma unroll
            for (int i = 0; i < m; ++i) b[j][k][i] = oL[((f * FP + k) * NB + 2 * u + i) * 32];
          }
          if constexpr (FT) {
            x8[j] = get_frag8(sFr + f * FS, FP, lane);
#pragma unroll
            for (int i = 0; i < m; ++i) b8[j][i] = oLt[(f * NB + 2 * u + i) * 32];
          }
        }
#pragma unroll
        for (int k = 0; k < FP; ++k)
          mma_pair2<PR, PR>(L[0], x[0][k], b[0][k], L[1], x[1][k], b[1][k], SET && k == 0, SET && k == 0);
        if constexpr (FT) mma_pair2<PR, PR>(L[0], x8[0], b8[0], L[1], x8[1], b8[1]);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int f = f0 + j;
            const float4 nn = *reinterpret_cast<const float4 *>(sGeo + (g + 8 * h) * 28 + 4 * f);
            const float s = sInv[f * 16 + g + 8 * h];
            const float nx = -nn.y * s, ny = -nn.z * s, nz = -nn.w * s;
#pragma unroll
            for (int i = 0; i < m; ++i)
#pragma unroll
              for (int v = 2 * h; v < 2 * h + 2; ++v) {
                const float l = L[j][i][v];
                rr[i][v] = fmaf(l, s, rr[i][v]);
                rv[0][i][v] = fmaf(l, nx, rv[0][i][v]);
                rv[1][i][v] = fmaf(l, ny, rv[1][i][v]);
                rv[2][i][v] = fmaf(l, nz, rv[2][i][v]);
              }
          }
      }
#pragma unroll
      for (int i = 0; i < m; ++i)
#pragma unroll
        for (int v = 0; v < 4; ++v) rr[i][v] = fmaf(rd[i][v], v < 2 ? uia : uib, rr[i][v]);
#pragma unroll
      for (int i = 0; i < m; ++i) {
        ma = fmaxf(ma, fmaxf(fabsf(rr[i][0]), fabsf(rr[i][1])));
        mb = fmaxf(mb, fmaxf(fabsf(rr[i][2]), fabsf(rr[i][3])));
#pragma unroll
        for (int v = 0; v < 4; ++v) r[i][v] = rr[i][v];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T y, q;
        Un::lsrk(ra[c], Un::row(rv[c], 0), xa[c], P, y, q);
        if (va) {
          Un::template store<Np, V>(Ra + (c + 1) * Np, n, y);
          Un::template store<Np, V>(Oa + (c + 1) * Np, n, q);
        }
        Un::lsrk(rb[c], Un::row(rv[c], 1), xb[c], P, y, q);
        if (vb) {
          Un::template store<Np, V>(Rb + (c + 1) * Np, n, y);
          Un::template store<Np, V>(Ob + (c + 1) * Np, n, q);
        }
      }
    };
    if (w < KP) {
      if constexpr (KP > 0) rhs_unit(std::integral_constant<int, 2>(), w, rp);
    } else {
      if constexpr (KT > 0) rhs_unit(std::integral_constant<int, 1>(), w, rp);
    }
    const float cma = __ldg(P.c2max + ka), cmb = __ldg(P.c2max + kb);
    ma = quad_max(ma), mb = quad_max(mb);
    if (t == 0) sMaxR[w * 16 + g] = ma, sMaxR[w * 16 + g + 8] = mb;
    group_sync<GW>(grp);  // maxima ready; operands, fluxes and geometry consumed

    // ---- 4. split rhs_p; the next tile on its way
    if (it + step < P.nit) fetch_tile(nshot, kn);
    float oia, oib, via, vib, da, db;
    {
      ma = sMaxR[g], mb = sMaxR[g + 8];
#pragma unroll
      for (int i = 1; i < GW; ++i) ma = fmaxf(ma, sMaxR[i * 16 + g]), mb = fmaxf(mb, sMaxR[i * 16 + g + 8]);
      const int sa = scale_field(ma), sb = scale_field(mb);
      const float ca = pow2_field(sa), cb = pow2_field(sb);
      via = pow2_field(254 - sa) * P.iV, vib = pow2_field(254 - sb) * P.iV;
      // |Vq r| c2 <= vnorm max|r| max c2 bounds the weighted cubature values
      const int wa = scale_field(P.vnorm * ma * cma),
                wb = scale_field(P.vnorm * mb * cmb);
      da = pow2_field(wa), db = pow2_field(wb);
      oia = pow2_field(254 - wa) * P.iP, oib = pow2_field(254 - wb) * P.iP;
      if (w < KP) Unit<2>::split(sR, w, lane, Unit<2>::row(rp, 0), Unit<2>::row(rp, 1), ca, cb);
      else
        Unit<1>::split(sR, w, lane, make_float2(rp[0][0], rp[0][1]), make_float2(rp[0][2], rp[0][3]), ca,
                       cb);
    }
    const float4 *Ca = reinterpret_cast<const float4 *>(P.c2p + (size_t)ka * P.Nq16) + t,
                 *Cb = reinterpret_cast<const float4 *>(P.c2p + (size_t)kb * P.Nq16) + t;
    const int nch = P.Nq16 / 16;
    group_sync<GW>(grp);  // rhs_p ready

    // residual of p: loaded here it is in flight during the projection, where
    // the registers allow (N = 7 187 -> 173 us per stage, N = 4 19.3 -> 19.7)
    float4 ra, rb;
    auto load_rp = [&]() {
      if (w < KP) {
        ra = load4<Np, V>(Ra, 16 * w + 4 * t), rb = load4<Np, V>(Rb, 16 * w + 4 * t);
      } else {
        const float2 x = load2<Np, V>(Ra, 16 * w + 2 * t), y = load2<Np, V>(Rb, 16 * w + 2 * t);
        ra = make_float4(x.x, x.y, 0.f, 0.f), rb = make_float4(y.x, y.y, 0.f, 0.f);
      }
    };
    if constexpr (C::EARLY) load_rp();

    // ---- 5. WADG projection of rhs_p, RC chunks of 16 cubature points at a
    //         time: Vq and c2 of the warp's chunks, then Pq of its unit
    float o[2][4] = {};
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += C::RC) {
      const int cend = min(nch, c0 + C::RC);
      if (c0 > 0) group_sync<GW>(grp);  // the last round's values are consumed
#pragma unroll 1
      for (int c = c0 + w; c < cend; c += GW) {
        const float4 za = __ldg(Ca + c * 4), zb = __ldg(Cb + c * 4);
        float v[2][4] = {};
        OpTile<uint4> bv[OPS ? 1 : KP][2];
        if constexpr (!OPS)
#pragma unroll
          for (int k = 0; k < KP; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i) bv[k][i] = oV[((c * KP + k) * 2 + i) * 32];
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          const Frag x = get_frag(sR, k, lane);
          const OpTile<uint4> b[2] = {OPS ? oV[((c * KP + k) * 2) * 32] : bv[OPS ? 0 : k][0],
                                      OPS ? oV[((c * KP + k) * 2 + 1) * 32] : bv[OPS ? 0 : k][1]};
          mma_tiles<PR>(v, x, b, SET && k == 0);
        }
        if constexpr (KT) {
          const Frag8 x = get_frag8(sR, KP, lane);
          const OpTile<uint2> b[2] = {oVt[(c * 2) * 32], oVt[(c * 2 + 1) * 32]};
          mma_tiles<PR>(v, x, b);
        }
        // points 16 c + 4 t + 0 .. 3 of the two rows
        const float4 xa = make_float4(v[0][0] * via * za.x, v[0][1] * via * za.y,
                                      v[1][0] * via * za.z, v[1][1] * via * za.w);
        const float4 xb = make_float4(v[0][2] * vib * zb.x, v[0][3] * vib * zb.y,
                                      v[1][2] * vib * zb.z, v[1][3] * vib * zb.w);
        Unit<2>::split(sW, c - c0, lane, xa, xb, da, db);
      }
      if constexpr (!OPS) {
        // operators from L2: the next four chunks' loads in flight
        OpTile<uint4> b[4][2];
        auto load_p = [&](int c) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i)
              b[j][i] = oP[(min(c + j, nch - 1) * NB + min(2 * w + i, NB - 1)) * 32];
        };
        load_p(c0);
        group_sync<GW>(grp);  // the round's values ready
#pragma unroll 1
        for (int c = c0; c < cend; c += 4) {
          OpTile<uint4> bb[4][2];
#pragma unroll
          for (int j = 0; j < 4; ++j) bb[j][0] = b[j][0], bb[j][1] = b[j][1];
          if (c + 4 < cend) load_p(c + 4);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (c + j >= cend) break;
            const Frag x = get_frag(sW, c + j - c0, lane);
            if (w < KP) mma_tiles<PR>(o, x, bb[j]);
            else mma_tile<PR>(o[0], x, bb[j][0]);
          }
        }
        continue;
      }
      group_sync<GW>(grp);  // the round's values ready
      constexpr int PU = PR == 4 ? 2 : 1;
#pragma unroll PU
      for (int c = c0; c < cend; ++c) {
        const Frag x = get_frag(sW, c - c0, lane);
        if (w < KP) {
          const OpTile<uint4> b[2] = {oP[(c * NB + 2 * w) * 32], oP[(c * NB + 2 * w + 1) * 32]};
          mma_tiles<PR>(o, x, b);
        } else {
          mma_tile<PR>(o[0], x, oP[(c * NB + 2 * w) * 32]);
        }
      }
    }

    // ---- 6. sources and the LSRK update of p
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) o[j][v] *= v < 2 ? oia : oib;
    if (P.src_tile)
      tile_sources(P, Np, shot, k0, [&](int e, float amp, const float *vec) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (w >= KP && j > 0) continue;
          const int n = w < KP ? 16 * w + 4 * t + 2 * j : 16 * KP + 2 * t;
          const float s0 = n < Np ? amp * __ldg(vec + n) : 0.f;
          const float s1 = n + 1 < Np ? amp * __ldg(vec + n + 1) : 0.f;
          if (e == g) o[j][0] += s0, o[j][1] += s1;
          if (e == g + 8) o[j][2] += s0, o[j][3] += s1;
        }
      });
    auto update_p = [&](auto M, int u, const float (&x)[2][4]) {
      using Un = Unit<decltype(M)::value>;
      using T = typename Un::T;
      const int n = Un::node(u, t);
      T pa, pb, fa, fb, sa, sb;
      if constexpr (!C::EARLY) {
        sa = Un::template load<Np, V>(Ra, n), sb = Un::template load<Np, V>(Rb, n);
      } else if constexpr (decltype(M)::value == 2) {
        sa = ra, sb = rb;
      } else {
        sa = lo2(ra), sb = lo2(rb);
      }
      if constexpr (decltype(M)::value == 2) {
        pa = qa[0], pb = qb[0];
      } else {
        pa = lo2(qa[0]), pb = lo2(qb[0]);
      }
      if constexpr (decltype(M)::value == 2) {
        fa = Un::row(x, 0), fb = Un::row(x, 1);
      } else {
        fa = make_float2(x[0][0], x[0][1]), fb = make_float2(x[0][2], x[0][3]);
      }
      T y, q;
      Un::lsrk(sa, fa, pa, P, y, q);
      if (va) {
        Un::template store<Np, V>(Ra, n, y);
        Un::template store<Np, V>(Oa, n, q);
      }
      Un::lsrk(sb, fb, pb, P, y, q);
      if (vb) {
        Un::template store<Np, V>(Rb, n, y);
        Un::template store<Np, V>(Ob, n, q);
      }
    };
    if (w < KP) {
      if constexpr (KP > 0) update_p(std::integral_constant<int, 2>(), w, o);
    } else {
      if constexpr (KT > 0) update_p(std::integral_constant<int, 1>(), w, o);
    }
  }
}

// ---------------------------------------------------------------- host side
template <int N>
static size_t group_smem(const WarpPlan &pl, int place) {
  using C = GroupCfg<N>;
  const int n = place == OPS_SHARED ? pl.ops_n : place == OPS_RESTS ? pl.ops_n - pl.oM : 0;
  return (size_t)n * 16 + (size_t)pl.table_ints * 4 + (size_t)C::NG * C::SCR * 4;
}

template <int N, int PR, int PLACE>
static bbw_status group_launch_as(const WarpPlan &pl, const WarpParams &P, int grid, cudaStream_t st) {
  using C = GroupCfg<N>;
  launch_stage_kernel(k_group_stage<N, PR, PLACE>, grid, C::T, group_smem<N>(pl, PLACE), st,
                      PLACE == OPS_SHARED && pl.chained, P);
  return check_launch("group-matrix stage");
}

// split FP16 contexts (three products) exist at N <= 5
template <int N>
static bbw_status group_launch_n(const WarpPlan &pl, const float *Qin, float *Qout, float *res,
                                 float fa, float fb, float fdt, float cstage, cudaStream_t st) {
  using C = GroupCfg<N>;
  WarpParams P = warp_params(pl, Qin, Qout, res, fa, fb, fdt, cstage);
  const int grid = warp_grid(pl, C::NG, P);
  if constexpr (C::OPS) {
    if (pl.products == 3)
      return pl.group_ops == OPS_SHARED ? group_launch_as<N, 3, OPS_SHARED>(pl, P, grid, st)
                                        : group_launch_as<N, 3, OPS_L2>(pl, P, grid, st);
    if (pl.group_ops == OPS_SHARED) return group_launch_as<N, 4, OPS_SHARED>(pl, P, grid, st);
  }
  return pl.group_ops == OPS_RESTS ? group_launch_as<N, 4, OPS_RESTS>(pl, P, grid, st)
                                   : group_launch_as<N, 4, OPS_L2>(pl, P, grid, st);
}

template <int N>
static bbw_status group_prepare_n(WarpPlan &pl) {
  using C = GroupCfg<N>;
  const size_t maxsm = (size_t)device_smem_optin();
  if (!C::OPS && pl.products == 3)
    return set_error(BBW_ERR_UNSUPPORTED, "group-matrix stage: three products at N <= 5 only");
  pl.group_ops = C::OPS && group_smem<N>(pl, OPS_SHARED) <= maxsm ? OPS_SHARED
                 : pl.products == 4 && group_smem<N>(pl, OPS_RESTS) <= maxsm ? OPS_RESTS : OPS_L2;
  if (group_smem<N>(pl, pl.group_ops) > maxsm)
    return set_error(BBW_ERR_UNSUPPORTED, "group-matrix stage: does not fit in shared memory");
  std::vector<const void *> fn = {(const void *)k_group_stage<N, 4, OPS_L2>,
                                  (const void *)k_group_stage<N, 4, OPS_RESTS>};
  if constexpr (C::OPS) {
    fn.push_back((const void *)k_group_stage<N, 4, OPS_SHARED>);
    fn.push_back((const void *)k_group_stage<N, 3, OPS_SHARED>);
    fn.push_back((const void *)k_group_stage<N, 3, OPS_L2>);
  }
  for (const void *f : fn) {
    const bbw_status s = ensure_smem_limit(f, (int)maxsm, "group-matrix stage attribute");
    if (s != BBW_OK) return s;
  }
  return BBW_OK;
}

#define BBW_GROUP_STAGE_INSTANCE(n)                                                             \
  bbw_status group_launch_##n(const WarpPlan &pl, const float *Qin, float *Qout, float *res,    \
                              float fa, float fb, float fdt, float cstage, cudaStream_t st) {   \
    return group_launch_n<n>(pl, Qin, Qout, res, fa, fb, fdt, cstage, st);                      \
  }                                                                                             \
  bbw_status group_prepare_##n(WarpPlan &pl) { return group_prepare_n<n>(pl); }

}  // namespace bbw
