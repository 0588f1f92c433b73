// One LSRK stage with every contraction on warp-level matrix instructions
// (mma.sync m16n8k16, FP16 pairs, FP32 accumulation).
//
// Replaces rk_volume + rk_surface + rk_update_WADG of the reference
// (cpp/okl/WaveKernels.okl:44-260, cpp/okl/WaveKernelsWADG.okl:1760-1887).
//
// A warp owns 16 elements from the trace gather to the LSRK update.  Elements
// are the rows (M = 16) of every product and operator rows the columns, so
// the accumulator of one contraction has the register layout of the next
// one's A operand: rhs_p -> Vq -> c2 -> Pq chains in registers, without
// shared memory, TMEM round trips or any barrier between warps.  The
// contractions are skinny (K = Np, Nfp or Nq <= 216 per element): what bounds
// them is the chain of dependent phases, not the tensor rate.  mma.sync gives
// 1024 FMA per cycle and SM here (8 cycles per m16n8k16 and SM quarter,
// measured), a quarter of what tcgen05 does on full tiles.
//
// FP32 values x are split into FP16 pairs x s = hi + lo with a power of two s
// per element and operand, so each element keeps its own dynamic range; the
// pair holds 23 bits.  With four products (hi hi, hi lo, lo hi, lo lo) the
// contraction error is that of FP32 sums; the split-FP16 form uses three.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "device_common.cuh"
#include "warp_stage.h"

namespace bbw {

struct WarpParams {
  int K, K0, Kc, Nq, Nq16, bc, pat_off, table_ints, nit, bs, ws, nt32;
  int oDt, oL, oLt, oV, oVt, oP, ops_n;  // operator offsets and size in uint4
  float fa, fb, fdt, cstage;
  float iD, iL, iV, iP, vnorm;      // inverse operator scales, max row sum of |Vq|
  const float *__restrict__ Qin;
  float *__restrict__ Qout;
  float *__restrict__ res;
  const float *__restrict__ geo;    // [K + 16][28]: fgeo 16 | vgeo 9 | pad
  const float *__restrict__ c2p;    // [K][Nq16], zero past Nq
  const float *__restrict__ c2max;
  const int *__restrict__ nbr;
  const int *__restrict__ tables;
  const uint4 *__restrict__ ops;
  const int *__restrict__ src_tile;
  const int *__restrict__ src_elem;
  const float *__restrict__ src_vec;
  float f0, tR, samp;
  const double *__restrict__ time;
};

template <int N>
struct WarpCfg {
  static constexpr int Np = NP(N), Nfp = NFP(N), EW = 4 * Np;
  // blocks of eight nodes: pairs of them are the k16 steps, an odd last one
  // is a k8 step (same for the face nodes)
  static constexpr int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2;
  static constexpr int FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  // the warps' state tiles in shared memory up to N = 5, the operators too
  // when they fit beside them (OPS); above, both through L1 / L2 and the
  // split face fluxes in shared memory instead of registers
  static constexpr bool SM = N <= 5;
  static constexpr bool FLUX_SM = N >= 6;
  // separate accumulators for the leading and the correction products
  static constexpr bool SEP = N <= 7;
#ifndef BBW_W3
#define BBW_W3 8
#endif
  static constexpr int W = N <= 2 ? 12 : N == 3 ? BBW_W3 : 8;  // warps per CTA
  static constexpr int T = 32 * W;
  static constexpr int V = Np % 4 == 0 ? 4 : Np % 2 == 0 ? 2 : 1;  // vector width of a row
  // state tile of a warp: rows of 4 Np floats, padded so that two rows of a
  // pair start 16 banks apart (a 16-byte access serves two rows at a time)
  static constexpr int ODD = V == 4 ? (48 - EW % 32) % 32 : 0;
  static constexpr int TILE = SM ? 16 * EW + 8 * ODD : 0;
  __host__ __device__ static constexpr int row(int e) { return e * EW + ((e + 1) >> 1) * ODD; }
  static constexpr int FLUX = 8 * FB * 8;                            // eight elements' fluxes
  static constexpr int FRAG = FLUX_SM ? 4 * (FP * 8 + FT * 4) * 32 : 0;
  static constexpr int RP = SM ? 0 : NB * 4 * 32;  // lifted part of rhs_p (SM: over p in the tile)
  static constexpr int SCR = TILE + FLUX + FRAG + RP;
};

__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                      uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// A operand of one k16 step: FP16 pairs of 16 elements x 16 columns.  Lane
// l holds elements l/4 (indices 0, 2) and l/4 + 8 (1, 3) at columns
// 4 (l%4) + {0, 1} (indices 0, 1) and + {2, 3}: the operators are packed with
// the matching column order, so four consecutive nodes sit in one lane.
struct Frag {
  uint32_t h[4], l[4];
};
struct Frag8 {  // a k8 step: columns 2 (l%4) + {0, 1}
  uint32_t h[2], l[2];
};

// x s = hi + lo for two values; s2 = (s, s)
__device__ __forceinline__ void split2(float2 x, float2 s2, uint32_t &h, uint32_t &l) {
  const float2 y = __fmul2_rn(x, s2);
  const __half2 hh = __float22half2_rn(y);
  const float2 f = __half22float2(hh);
  const __half2 ll = __float22half2_rn(__fadd2_rn(y, make_float2(-f.x, -f.y)));
  h = *reinterpret_cast<const uint32_t *>(&hh);
  l = *reinterpret_cast<const uint32_t *>(&ll);
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }
// LSRK update of two values: r = fa r + fdt x (returned), q += fb r
__device__ __forceinline__ float2 lsrk2(float2 r, float2 x, float2 fa, float2 fdt) {
  return __ffma2_rn(fa, r, __fmul2_rn(fdt, x));
}
// rows a (elements l/4) and b (l/4 + 8), scaled by ca and cb
__device__ __forceinline__ void split_frag(Frag &f, const float4 a, const float4 b, float ca,
                                           float cb) {
  split2(lo2(a), both(ca), f.h[0], f.l[0]);
  split2(lo2(b), both(cb), f.h[1], f.l[1]);
  split2(hi2(a), both(ca), f.h[2], f.l[2]);
  split2(hi2(b), both(cb), f.h[3], f.l[3]);
}
__device__ __forceinline__ void split_frag(Frag8 &f, const float2 a, const float2 b, float ca,
                                           float cb) {
  split2(a, both(ca), f.h[0], f.l[0]);
  split2(b, both(cb), f.h[1], f.l[1]);
}

// leading products into c, corrections into e (the same array, or its own so
// that the small terms add up before they meet the large ones: the matrix
// unit's sums round toward zero, so fewer large sums leave less bias)
template <int PR>
__device__ __forceinline__ void mma_tile(float (&c)[4], float (&e)[4], const Frag &x,
                                         const uint4 b) {
  mma16(c, x.h, b.x, b.y);
  mma16(e, x.h, b.z, b.w);
  mma16(e, x.l, b.x, b.y);
  if constexpr (PR == 4) mma16(e, x.l, b.z, b.w);
}
template <int PR, int M>
__device__ __forceinline__ void mma_tiles(float (&c)[M][4], float (&e)[M][4], const Frag &x,
                                          const uint4 (&b)[M]) {
#pragma unroll
  for (int i = 0; i < M; ++i) mma16(c[i], x.h, b[i].x, b[i].y);
#pragma unroll
  for (int i = 0; i < M; ++i) mma16(e[i], x.h, b[i].z, b[i].w);
#pragma unroll
  for (int i = 0; i < M; ++i) mma16(e[i], x.l, b[i].x, b[i].y);
  if constexpr (PR == 4) {
#pragma unroll
    for (int i = 0; i < M; ++i) mma16(e[i], x.l, b[i].z, b[i].w);
  }
}
template <int PR, int M>
__device__ __forceinline__ void mma_tiles(float (&c)[M][4], float (&e)[M][4], const Frag8 &x,
                                          const uint2 (&b)[M]) {
#pragma unroll
  for (int i = 0; i < M; ++i) mma8(c[i], x.h[0], x.h[1], b[i].x);
#pragma unroll
  for (int i = 0; i < M; ++i) mma8(e[i], x.h[0], x.h[1], b[i].y);
#pragma unroll
  for (int i = 0; i < M; ++i) mma8(e[i], x.l[0], x.l[1], b[i].x);
  if constexpr (PR == 4) {
#pragma unroll
    for (int i = 0; i < M; ++i) mma8(e[i], x.l[0], x.l[1], b[i].y);
  }
}

// power of two that brings a maximum m below 2^15, as an exponent field; the
// inverse is the field 254 - f.  Clamped so that both stay normal numbers
// (m below 2^-99, zero included, takes 2^113).
__device__ __forceinline__ int scale_field(float m) {
  const int e = (int)((__float_as_uint(m) >> 23) & 255u);
  return min(max(268 - e, 14), 240);
}
__device__ __forceinline__ float pow2_field(int f) { return __uint_as_float((uint32_t)f << 23); }

// maximum over the four lanes that share an element row
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float max4(float m, const float4 v) {
  return fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
}
__device__ __forceinline__ float max2(float m, const float2 v) {
  return fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
}

// x[n .. n+3] (n a multiple of 4) and x[n .. n+1] (n even) of a row of LEN
// values, zero past its end; V: widest aligned access
template <int LEN, int V>
__device__ __forceinline__ float4 load4(const float *x, int n) {
  if constexpr (V == 4) {
    return n < LEN ? *reinterpret_cast<const float4 *>(x + n) : make_float4(0.f, 0.f, 0.f, 0.f);
  } else if constexpr (V == 2) {
    const float2 z = make_float2(0.f, 0.f);
    const float2 a = n < LEN ? *reinterpret_cast<const float2 *>(x + n) : z;
    const float2 b = n + 2 < LEN ? *reinterpret_cast<const float2 *>(x + n + 2) : z;
    return make_float4(a.x, a.y, b.x, b.y);
  } else {
    return make_float4(n < LEN ? x[n] : 0.f, n + 1 < LEN ? x[n + 1] : 0.f,
                       n + 2 < LEN ? x[n + 2] : 0.f, n + 3 < LEN ? x[n + 3] : 0.f);
  }
}
template <int LEN, int V>
__device__ __forceinline__ float2 load2(const float *x, int n) {
  if constexpr (V >= 2) {
    return n < LEN ? *reinterpret_cast<const float2 *>(x + n) : make_float2(0.f, 0.f);
  } else {
    return make_float2(n < LEN ? x[n] : 0.f, n + 1 < LEN ? x[n + 1] : 0.f);
  }
}
template <int LEN, int V>
__device__ __forceinline__ void store4(float *x, int n, const float4 v) {
  if constexpr (V == 4) {
    if (n < LEN) *reinterpret_cast<float4 *>(x + n) = v;
  } else if constexpr (V == 2) {
    if (n < LEN) *reinterpret_cast<float2 *>(x + n) = make_float2(v.x, v.y);
    if (n + 2 < LEN) *reinterpret_cast<float2 *>(x + n + 2) = make_float2(v.z, v.w);
  } else {
    if (n < LEN) x[n] = v.x;
    if (n + 1 < LEN) x[n + 1] = v.y;
    if (n + 2 < LEN) x[n + 2] = v.z;
    if (n + 3 < LEN) x[n + 3] = v.w;
  }
}
template <int LEN, int V>
__device__ __forceinline__ void store2(float *x, int n, const float2 v) {
  if constexpr (V >= 2) {
    if (n < LEN) *reinterpret_cast<float2 *>(x + n) = v;
  } else {
    if (n < LEN) x[n] = v.x;
    if (n + 1 < LEN) x[n + 1] = v.y;
  }
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Ricker wavelet amp (1 - 2 a^2) exp(-a^2), a = pi f0 (t - tR)
__device__ __forceinline__ float warp_ricker(float t, float f0, float tR, float amp) {
  const float a = 3.14159265358979f * f0 * (t - tR);
  return amp * (1.f - 2.f * a * a) * expf(-a * a);
}

// bulk L2 prefetch of [p, p + bytes), trimmed to 16-byte boundaries
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
  const size_t a = (reinterpret_cast<size_t>(p) + 15) & ~(size_t)15;
  const size_t e = (reinterpret_cast<size_t>(p) + bytes) & ~(size_t)15;
  if (e > a)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(a), "r"((uint32_t)(e - a)));
}

// Gather of face f of eight elements h8 .. h8 + 7 of the warp's tile, nodes
// I0 .. I0 + NI - 1: EPI elements per pass, lane = (element, node), so a pass
// reads the face nodes of a neighbour's row together.
template <int N, int I0, int NI>
struct FaceGather {
  using C = WarpCfg<N>;
  static constexpr int EPI = NI >= 32 ? 1 : (32 / NI > 8 ? 8 : 32 / NI);
  static constexpr int IT = (8 + EPI - 1) / EPI;
  float X[IT][4];
  float4 g[IT];
  uint32_t walls;

  __device__ __forceinline__ static int sub(int lane) { return lane / NI < EPI ? lane / NI : 0; }
  __device__ __forceinline__ static int node(int lane) {
    return lane / NI < EPI ? I0 + lane % NI : I0;
  }
  __device__ __forceinline__ static int elem(int it, int lane) {
    const int e = it * EPI + sub(lane);
    return IT * EPI > 8 && it == IT - 1 ? min(e, 7) : e;
  }

  // code: neighbour codes of the tile's faces, one per lane ((element % 8) * 4
  // + face) for this half
  __device__ __forceinline__ void load(const WarpParams &P, const float *__restrict__ Qs,
                                       const float *sQ, const int *sFm, const int *sPat, int f,
                                       int h8, int k0, int klast, int code, int lane) {
    const int i = node(lane), own = sFm[f * C::Nfp + i];
    const float4 *geo = reinterpret_cast<const float4 *>(P.geo) + (size_t)(k0 + h8) * 7 + f;
    walls = 0;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = elem(it, lane);
      const int cd = __shfl_sync(0xffffffffu, code, e * 4 + f);
      const int pat = cd & 255;
      const bool wall = pat == 255;
      walls |= wall ? 1u << it : 0u;
      const int nn = wall ? own : sPat[pat * C::Nfp + i];
      const float *x = Qs + (size_t)(cd >> 8) * C::EW + nn;
#pragma unroll
      for (int c = 0; c < 4; ++c) X[it][c] = __ldg(x + c * C::Np);
      g[it] = __ldg(geo + e * 7);
    }
  }
  // upwind pressure flux to sF[element][8 FB].  A wall's + trace is the own
  // one with the pressure (p = 0 wall) or the velocity (rigid) reversed.
  __device__ __forceinline__ void flux(const WarpParams &P, const float *__restrict__ Qs,
                                       const float *sQ, const int *sFm, float *sF, int f, int h8,
                                       int k0, int klast, int lane) const {
    const bool act = lane / NI < EPI;
    const int i = node(lane), own = sFm[f * C::Nfp + i];
    const float wp = P.bc == BBW_BC_PRESSURE_RELEASE ? -1.f : 1.f, wu = -wp;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = elem(it, lane);
      const float *m = C::SM ? sQ + C::row(h8 + e) + own
                             : Qs + (size_t)min(k0 + h8 + e, klast) * C::EW + own;
      const bool wall = walls >> it & 1u;
      const float sp = wall ? wp : 1.f, su = wall ? wu : 1.f;
      const float dp = fmaf(sp, X[it][0], -m[0]);
      float un = fmaf(su, X[it][1], -m[C::Np]) * g[it].y;
      un = fmaf(fmaf(su, X[it][2], -m[2 * C::Np]), g[it].z, un);
      un = fmaf(fmaf(su, X[it][3], -m[3 * C::Np]), g[it].w, un);
      const float fl = .5f * g[it].x * (dp - un);
      if (IT * EPI > 8 && it == IT - 1) {
        if (act && it * EPI + sub(lane) < 8) sF[e * (8 * C::FB) + i] = fl;
      } else {
        if (act) sF[e * (8 * C::FB) + i] = fl;
      }
    }
  }
};

template <int N, bool WIDE>
struct HalfFace;
template <int N>
struct HalfFace<N, false> {
  FaceGather<N, 0, NFP(N)> a;
  template <class... A>
  __device__ __forceinline__ void load(A... x) { a.load(x...); }
  template <class... A>
  __device__ __forceinline__ void flux(A... x) const { a.flux(x...); }
};
template <int N>
struct HalfFace<N, true> {  // more than 32 nodes per face
  FaceGather<N, 0, 32> a;
  FaceGather<N, 32, (NFP(N) > 32 ? NFP(N) - 32 : 1)> b;
  template <class... A>
  __device__ __forceinline__ void load(A... x) { a.load(x...), b.load(x...); }
  template <class... A>
  __device__ __forceinline__ void flux(A... x) const { a.flux(x...), b.flux(x...); }
};

// res = fa res + fdt rhs, Q += fb res for four values
__device__ __forceinline__ void lsrk4(const float4 r0, const float4 x, const float4 q0,
                                      const WarpParams &P, float4 &r, float4 &q) {
  const float2 a = lsrk2(lo2(r0), lo2(x), both(P.fa), both(P.fdt));
  const float2 b = lsrk2(hi2(r0), hi2(x), both(P.fa), both(P.fdt));
  const float2 c = __ffma2_rn(both(P.fb), a, lo2(q0)), d = __ffma2_rn(both(P.fb), b, hi2(q0));
  r = make_float4(a.x, a.y, b.x, b.y), q = make_float4(c.x, c.y, d.x, d.y);
}

template <int N, int PR, bool OPS>
__global__ void __launch_bounds__(WarpCfg<N>::T, 1) k_warp_stage(const WarpParams P) {
  using C = WarpCfg<N>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW;
  constexpr int FB = C::FB, FP = C::FP, FT = C::FT, V = C::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  uint4 *sOps = reinterpret_cast<uint4 *>(smem_raw);
  const int nops = OPS ? P.ops_n : 0;
  int *sTab = reinterpret_cast<int *>(sOps + nops);
  float *scr = reinterpret_cast<float *>(sTab + P.table_ints) + warp * C::SCR;
  if constexpr (OPS)
    for (int i = tid; i < P.ops_n; i += C::T) sOps[i] = __ldg(P.ops + i);
  for (int i = tid; i < P.table_ints; i += C::T) sTab[i] = __ldg(P.tables + i);
  float *sQ = scr, *sF = scr + C::TILE;
  uint4 *sFr = reinterpret_cast<uint4 *>(sF + C::FLUX);
  float *sRp = sF + C::FLUX + C::FRAG;
  if constexpr (FB * 8 > Nfp)  // flux columns past Nfp meet zero operator columns
    for (int i = lane; i < C::FLUX; i += 32) sF[i] = 0.f;
  __syncthreads();
  const uint4 *ops = OPS ? sOps : P.ops;
  const uint4 *oD = ops + lane, *oL = ops + P.oL + lane, *oV = ops + P.oV + lane,
              *oP = ops + P.oP + lane;
  const uint2 *oDt = reinterpret_cast<const uint2 *>(ops + P.oDt) + lane,
              *oLt = reinterpret_cast<const uint2 *>(ops + P.oLt) + lane,
              *oVt = reinterpret_cast<const uint2 *>(ops + P.oVt) + lane;
  const int *sPat = sTab + P.pat_off;
  const int ntile = (P.Kc - P.K0 + 15) / 16, klast = P.Kc - 1;
  const size_t shot_stride = (size_t)P.K * EW;
  const int step = gridDim.x * C::W;

  // state tile of item i to shared memory; neighbour codes of its faces
  auto fetch_tile = [&](int i) {
    const int sh = i / ntile, kn = P.K0 + (i - sh * ntile) * 16, ne = min(16, P.Kc - kn);
    const float *src = P.Qin + sh * shot_stride + (size_t)kn * EW;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sQ);
#pragma unroll 4
    for (int e = 0; e < ne; ++e)
#pragma unroll
      for (int c = 0; c < Np; c += 32)
        if (c + lane < Np)
          cp_async16(dst + 4 * (C::row(e) + 4 * (c + lane)),
                     src + e * EW + 4 * (c + lane));
  };
  auto codes = [&](int i, int &c0, int &c1) {
    const int sh = i / ntile, kn = P.K0 + (i - sh * ntile) * 16;
    c0 = __ldg(P.nbr + (size_t)min(kn + g, klast) * 4 + t);
    c1 = __ldg(P.nbr + (size_t)min(kn + 8 + g, klast) * 4 + t);
  };

  int it = blockIdx.x * P.bs + warp * P.ws;
  int code0 = 0, code1 = 0;
  if (it < P.nit) {
    if constexpr (C::SM) fetch_tile(it);
    codes(it, code0, code1);
  }
  for (; it < P.nit; it += step) {
    const int shot = it / ntile, k0 = P.K0 + (it - shot * ntile) * 16;
    const float *Qs = P.Qin + shot * shot_stride;
    const int ka = min(k0 + g, klast), kb = min(k0 + g + 8, klast);
    const bool va = k0 + g < P.Kc, vb = k0 + g + 8 < P.Kc;
    const size_t ea = (size_t)ka * EW, eb = (size_t)kb * EW;
    const float *Qa = C::SM ? sQ + C::row(ka - k0) : Qs + ea;
    const float *Qb = C::SM ? sQ + C::row(kb - k0) : Qs + eb;
    float *Ra = P.res + shot * shot_stride + ea, *Rb = P.res + shot * shot_stride + eb;
    float *Oa = P.Qout + shot * shot_stride + ea, *Ob = P.Qout + shot * shot_stride + eb;

    if (lane == 0) {  // the next item's inputs on their way to L2
      const int nx = it + step;
      if (nx < P.nit) {
        const int sh = nx / ntile, kn = P.K0 + (nx - sh * ntile) * 16, ne = min(16, P.Kc - kn);
        const size_t at = sh * shot_stride + (size_t)kn * EW;
        prefetch_l2(P.Qin + at, (size_t)ne * EW * 4);
        prefetch_l2(P.res + at, (size_t)ne * EW * 4);
        prefetch_l2(P.c2p + (size_t)kn * P.Nq16, (size_t)ne * P.Nq16 * 4);
      }
    }
    if constexpr (C::SM) cp_async_wait();
    __syncwarp();

    // ---- 1. face fluxes of eight elements at a time (the rows l/4, then
    //         l/4 + 8); the next half face's gather is in flight meanwhile
    Frag ff[C::FLUX_SM ? 1 : 4][FP > 0 && !C::FLUX_SM ? FP : 1];
    Frag8 f8[C::FLUX_SM ? 1 : 4];
    float fia[4], fib[4];  // inverse scales of the faces
    {
      HalfFace<N, (Nfp > 32)> buf[2];
      buf[0].load(P, Qs, sQ, sTab, sPat, 0, 0, k0, klast, code0, lane);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int f = r >> 1, h = r & 1;
        if (r < 7)
          buf[(r + 1) & 1].load(P, Qs, sQ, sTab, sPat, (r + 1) >> 1, 8 * ((r + 1) & 1), k0, klast,
                                (r + 1) & 1 ? code1 : code0, lane);
        buf[r & 1].flux(P, Qs, sQ, sTab, sF, f, 8 * h, k0, klast, lane);
        __syncwarp();
        const float *row = sF + g * (8 * FB);
        float4 x[FP > 0 ? FP : 1];
        float2 y = make_float2(0.f, 0.f);
        float m = 0.f;
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          x[k] = *reinterpret_cast<const float4 *>(row + 16 * k + 4 * t);
          m = max4(m, x[k]);
        }
        if constexpr (FT) {
          y = *reinterpret_cast<const float2 *>(row + 16 * FP + 2 * t);
          m = max2(m, y);
        }
        const int sc = scale_field(quad_max(m));
        const float cs = pow2_field(sc), inv = pow2_field(254 - sc) * P.iL;
        if (h == 0) fia[f] = inv;
        else fib[f] = inv;
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          uint32_t h0, h1, l0, l1;
          split2(lo2(x[k]), both(cs), h0, l0);
          split2(hi2(x[k]), both(cs), h1, l1);
          if constexpr (C::FLUX_SM) {  // (face, step): hi words of 32 lanes, then lo words
            uint32_t *d = reinterpret_cast<uint32_t *>(sFr + (f * FP + k) * 64);
            d[lane * 4 + h] = h0, d[lane * 4 + 2 + h] = h1;
            d[128 + lane * 4 + h] = l0, d[128 + lane * 4 + 2 + h] = l1;
          } else {
            ff[f][k].h[h] = h0, ff[f][k].h[2 + h] = h1;
            ff[f][k].l[h] = l0, ff[f][k].l[2 + h] = l1;
          }
        }
        if constexpr (FT) {
          uint32_t h0, l0;
          split2(y, both(cs), h0, l0);
          if constexpr (C::FLUX_SM) {
            uint32_t *d = reinterpret_cast<uint32_t *>(sFr + 4 * FP * 64 + f * 32);
            d[lane * 4 + h] = h0, d[lane * 4 + 2 + h] = l0;
          } else {
            f8[f].h[h] = h0, f8[f].l[h] = l0;
          }
        }
        __syncwarp();
      }
    }
    if (it + step < P.nit) codes(it + step, code0, code1);

    // ---- 2. pressure gradient, lift, and the update of u, v, w, 16 nodes at a
    //         time; the lifted part of rhs_p waits in shared memory (over p)
    float Ga[9], Gb[9], na[4][3], nb[4][3];
    {
      const float4 *A = reinterpret_cast<const float4 *>(P.geo) + (size_t)(k0 + g) * 7,
                   *B = A + 8 * 7;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const float4 x = __ldg(A + f), y = __ldg(B + f);
        // normals times the inverse scale of the face's flux
        na[f][0] = x.y * fia[f], na[f][1] = x.z * fia[f], na[f][2] = x.w * fia[f];
        nb[f][0] = y.y * fib[f], nb[f][1] = y.z * fib[f], nb[f][2] = y.w * fib[f];
      }
      const float4 a0 = __ldg(A + 4), a1 = __ldg(A + 5), a2 = __ldg(A + 6);
      const float4 b0 = __ldg(B + 4), b1 = __ldg(B + 5), b2 = __ldg(B + 6);
      Ga[0] = a0.x, Ga[1] = a0.y, Ga[2] = a0.z, Ga[3] = a0.w, Ga[4] = a1.x, Ga[5] = a1.y;
      Ga[6] = a1.z, Ga[7] = a1.w, Ga[8] = a2.x;
      Gb[0] = b0.x, Gb[1] = b0.y, Gb[2] = b0.z, Gb[3] = b0.w, Gb[4] = b1.x, Gb[5] = b1.y;
      Gb[6] = b1.z, Gb[7] = b1.w, Gb[8] = b2.x;
    }
    float Ma = 0.f, Mb = 0.f;  // bound of the contravariant velocities
    {
      Frag fp[KP > 0 ? KP : 1];
      Frag8 fp8;
      float pia, pib;
      {
        float4 xa[KP > 0 ? KP : 1], xb[KP > 0 ? KP : 1];
        float2 ya = make_float2(0.f, 0.f), yb = ya;
        float ma = 0.f, mb = 0.f;
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          xa[k] = load4<Np, V>(Qa, 16 * k + 4 * t), xb[k] = load4<Np, V>(Qb, 16 * k + 4 * t);
          ma = max4(ma, xa[k]), mb = max4(mb, xb[k]);
        }
        if constexpr (KT) {
          ya = load2<Np, V>(Qa, 16 * KP + 2 * t), yb = load2<Np, V>(Qb, 16 * KP + 2 * t);
          ma = max2(ma, ya), mb = max2(mb, yb);
        }
        const int sa = scale_field(quad_max(ma)), sb = scale_field(quad_max(mb));
        const float ca = pow2_field(sa), cb = pow2_field(sb);
        // minus the inverse scale, folded into the geometric factors below
        pia = -pow2_field(254 - sa) * P.iD, pib = -pow2_field(254 - sb) * P.iD;
#pragma unroll
        for (int k = 0; k < KP; ++k) split_frag(fp[k], xa[k], xb[k], ca, cb);
        if constexpr (KT) split_frag(fp8, ya, yb, ca, cb);
      }
      __syncwarp();
      float Ha[9], Hb[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) Ha[c] = Ga[c] * pia, Hb[c] = Gb[c] * pib;
      // one block of eight nodes: rhs of u, v, w and the lifted part of rhs_p
      auto block = [&](int j, float (&rv)[3][4], float (&rp)[4]) {
        {
          float d[3][4] = {}, e[3][4] = {};
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            uint4 b[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = oD[((c * KP + k) * NB + j) * 32];
            if constexpr (C::SEP) mma_tiles<PR>(d, e, fp[k], b);
            else mma_tiles<PR>(d, d, fp[k], b);
          }
          if constexpr (KT) {
            uint2 b[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = oDt[(c * NB + j) * 32];
            if constexpr (C::SEP) mma_tiles<PR>(d, e, fp8, b);
            else mma_tiles<PR>(d, d, fp8, b);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const bool lo = v < 2;
            const float *G = lo ? Ha : Hb;
            const float a = d[0][v] + e[0][v], b = d[1][v] + e[1][v], c = d[2][v] + e[2][v];
#pragma unroll
            for (int x = 0; x < 3; ++x) rv[x][v] = G[x] * a + G[3 + x] * b + G[6 + x] * c;
          }
        }
        // corrections of all steps first, then the leading products
        float L[4][4] = {};
        if constexpr (C::FLUX_SM) {
#pragma unroll
          for (int k = 0; k < FP; ++k)
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              const uint4 b = oL[((f * FP + k) * NB + j) * 32];
              const uint4 xh = sFr[(f * FP + k) * 64 + lane], xl = sFr[(f * FP + k) * 64 + 32 + lane];
              const Frag x = {{xh.x, xh.y, xh.z, xh.w}, {xl.x, xl.y, xl.z, xl.w}};
              mma_tile<PR>(L[f], L[f], x, b);
            }
          if constexpr (FT) {
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              const uint2 b = oLt[(f * NB + j) * 32];
              const uint4 q = sFr[4 * FP * 64 + f * 32 + lane];
              mma8(L[f], q.x, q.y, b.x);
              mma8(L[f], q.x, q.y, b.y);
              mma8(L[f], q.z, q.w, b.x);
              if constexpr (PR == 4) mma8(L[f], q.z, q.w, b.y);
            }
          }
        } else {
          uint4 b[FP > 0 ? FP : 1][4];
          uint2 c[4];
#pragma unroll
          for (int k = 0; k < FP; ++k)
#pragma unroll
            for (int f = 0; f < 4; ++f) b[k][f] = oL[((f * FP + k) * NB + j) * 32];
          if constexpr (FT) {
#pragma unroll
            for (int f = 0; f < 4; ++f) c[f] = oLt[(f * NB + j) * 32];
          }
#pragma unroll
          for (int k = 0; k < FP; ++k) {
            if constexpr (PR == 4) {
#pragma unroll
              for (int f = 0; f < 4; ++f) mma16(L[f], ff[f][k].l, b[k][f].z, b[k][f].w);
            }
#pragma unroll
            for (int f = 0; f < 4; ++f) mma16(L[f], ff[f][k].h, b[k][f].z, b[k][f].w);
#pragma unroll
            for (int f = 0; f < 4; ++f) mma16(L[f], ff[f][k].l, b[k][f].x, b[k][f].y);
          }
          if constexpr (FT) {
            if constexpr (PR == 4) {
#pragma unroll
              for (int f = 0; f < 4; ++f) mma8(L[f], f8[f].l[0], f8[f].l[1], c[f].y);
            }
#pragma unroll
            for (int f = 0; f < 4; ++f) mma8(L[f], f8[f].h[0], f8[f].h[1], c[f].y);
#pragma unroll
            for (int f = 0; f < 4; ++f) mma8(L[f], f8[f].l[0], f8[f].l[1], c[f].x);
#pragma unroll
            for (int f = 0; f < 4; ++f) mma8(L[f], f8[f].h[0], f8[f].h[1], c[f].x);
          }
#pragma unroll
          for (int k = 0; k < FP; ++k)
#pragma unroll
            for (int f = 0; f < 4; ++f) mma16(L[f], ff[f][k].h, b[k][f].x, b[k][f].y);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const bool lo = v < 2;
          rp[v] = 0.f;
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            rp[v] = fmaf(L[f][v], lo ? fia[f] : fib[f], rp[v]);
#pragma unroll
            for (int x = 0; x < 3; ++x) rv[x][v] = fmaf(-(lo ? na[f][x] : nb[f][x]), L[f][v], rv[x][v]);
          }
        }
      };
      float mu[3] = {0.f, 0.f, 0.f}, mv[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
      for (int k = 0; k < KP; ++k) {
        const int n = 16 * k + 4 * t;
        float4 ra[3], rb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          ra[c] = load4<Np, V>(Ra + (c + 1) * Np, n), rb[c] = load4<Np, V>(Rb + (c + 1) * Np, n);
        float x[3][4], y[3][4], px[4], py[4];
        block(2 * k, x, px);
        block(2 * k + 1, y, py);
        if constexpr (C::SM) {
          // row a: nodes n .. n + 3 of the lane's own slot in the p rows
          if (va) store4<Np, V>(const_cast<float *>(Qa), n, make_float4(px[0], px[1], py[0], py[1]));
          if (vb) store4<Np, V>(const_cast<float *>(Qb), n, make_float4(px[2], px[3], py[2], py[3]));
        } else {
          float4 *d = reinterpret_cast<float4 *>(sRp) + 2 * k * 32 + lane;
          d[0] = make_float4(px[0], px[1], py[0], py[1]);
          d[32] = make_float4(px[2], px[3], py[2], py[3]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float4 qa = load4<Np, V>(Qa + (c + 1) * Np, n), qb = load4<Np, V>(Qb + (c + 1) * Np, n);
          mu[c] = max4(mu[c], qa), mv[c] = max4(mv[c], qb);
          float4 r, q;
          lsrk4(ra[c], make_float4(x[c][0], x[c][1], y[c][0], y[c][1]), qa, P, r, q);
          if (va) {
            store4<Np, V>(Ra + (c + 1) * Np, n, r);
            store4<Np, V>(Oa + (c + 1) * Np, n, q);
          }
          lsrk4(rb[c], make_float4(x[c][2], x[c][3], y[c][2], y[c][3]), qb, P, r, q);
          if (vb) {
            store4<Np, V>(Rb + (c + 1) * Np, n, r);
            store4<Np, V>(Ob + (c + 1) * Np, n, q);
          }
        }
      }
      if constexpr (KT) {
        const int n = 16 * KP + 2 * t;
        float2 ra[3], rb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          ra[c] = load2<Np, V>(Ra + (c + 1) * Np, n), rb[c] = load2<Np, V>(Rb + (c + 1) * Np, n);
        float x[3][4], px[4];
        block(2 * KP, x, px);
        if constexpr (C::SM) {
          if (va) store2<Np, V>(const_cast<float *>(Qa), n, make_float2(px[0], px[1]));
          if (vb) store2<Np, V>(const_cast<float *>(Qb), n, make_float2(px[2], px[3]));
        } else {
          reinterpret_cast<float4 *>(sRp)[2 * KP * 32 + lane] = make_float4(px[0], px[1], px[2], px[3]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float2 qa = load2<Np, V>(Qa + (c + 1) * Np, n), qb = load2<Np, V>(Qb + (c + 1) * Np, n);
          mu[c] = max2(mu[c], qa), mv[c] = max2(mv[c], qb);
          const float2 r = make_float2(P.fa * ra[c].x + P.fdt * x[c][0], P.fa * ra[c].y + P.fdt * x[c][1]);
          const float2 s = make_float2(P.fa * rb[c].x + P.fdt * x[c][2], P.fa * rb[c].y + P.fdt * x[c][3]);
          if (va) {
            store2<Np, V>(Ra + (c + 1) * Np, n, r);
            store2<Np, V>(Oa + (c + 1) * Np, n, make_float2(qa.x + P.fb * r.x, qa.y + P.fb * r.y));
          }
          if (vb) {
            store2<Np, V>(Rb + (c + 1) * Np, n, s);
            store2<Np, V>(Ob + (c + 1) * Np, n, make_float2(qb.x + P.fb * s.x, qb.y + P.fb * s.y));
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) mu[c] = quad_max(mu[c]), mv[c] = quad_max(mv[c]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Ma = fmaxf(Ma, fabsf(Ga[3 * c]) * mu[0] + fabsf(Ga[3 * c + 1]) * mu[1] +
                           fabsf(Ga[3 * c + 2]) * mu[2]);
        Mb = fmaxf(Mb, fabsf(Gb[3 * c]) * mv[0] + fabsf(Gb[3 * c + 1]) * mv[1] +
                           fabsf(Gb[3 * c + 2]) * mv[2]);
      }
    }

    // ---- 3. divergence of the contravariant velocities
    float r[NB][4];
    {
      float e[C::SEP ? NB : 1][4];
      // twice the bound: its own rounding cannot bring a value to 2^16
      const int sa = scale_field(2.f * Ma), sb = scale_field(2.f * Mb);
      const float ca = pow2_field(sa), cb = pow2_field(sb);
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          r[j][v] = 0.f;
          if constexpr (C::SEP) e[j][v] = 0.f;
        }
      // products of one operand step with the tiles b of all node blocks
      auto accumulate = [&](const auto &u, const auto *B) {
        using T = std::remove_const_t<std::remove_reference_t<decltype(*B)>>;
#pragma unroll
        for (int j0 = 0; j0 < NB; j0 += 4) {
          constexpr int full = NB / 4 * 4, rem = NB % 4 ? NB % 4 : 4;
          if (j0 < full) {
            T b[4];
            float(&rr)[4][4] = *reinterpret_cast<float(*)[4][4]>(&r[j0]);
            float(&ee)[4][4] = *reinterpret_cast<float(*)[4][4]>(C::SEP ? &e[C::SEP ? j0 : 0] : &r[j0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(rr, ee, u, b);
          } else {
            T b[rem];
            float(&rr)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(&r[j0]);
            float(&ee)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(C::SEP ? &e[C::SEP ? j0 : 0] : &r[j0]);
#pragma unroll
            for (int j = 0; j < rem; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(rr, ee, u, b);
          }
        }
      };
#pragma unroll 1
      for (int k = 0; k < KP; ++k) {
        float4 xa[3], xb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xa[c] = load4<Np, V>(Qa + (c + 1) * Np, 16 * k + 4 * t);
          xb[c] = load4<Np, V>(Qb + (c + 1) * Np, 16 * k + 4 * t);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          auto con = [](const float4 (&x)[3], const float *G) {
            return make_float4(x[0].x * G[0] + x[1].x * G[1] + x[2].x * G[2],
                               x[0].y * G[0] + x[1].y * G[1] + x[2].y * G[2],
                               x[0].z * G[0] + x[1].z * G[1] + x[2].z * G[2],
                               x[0].w * G[0] + x[1].w * G[1] + x[2].w * G[2]);
          };
          Frag u;
          split_frag(u, con(xa, Ga + 3 * c), con(xb, Gb + 3 * c), ca, cb);
          accumulate(u, oD + (c * KP + k) * NB * 32);
        }
      }
      if constexpr (KT) {
        float2 xa[3], xb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xa[c] = load2<Np, V>(Qa + (c + 1) * Np, 16 * KP + 2 * t);
          xb[c] = load2<Np, V>(Qb + (c + 1) * Np, 16 * KP + 2 * t);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          auto con = [](const float2 (&x)[3], const float *G) {
            return make_float2(x[0].x * G[0] + x[1].x * G[1] + x[2].x * G[2],
                               x[0].y * G[0] + x[1].y * G[1] + x[2].y * G[2]);
          };
          Frag8 u;
          split_frag(u, con(xa, Ga + 3 * c), con(xb, Gb + 3 * c), ca, cb);
          accumulate(u, oDt + c * NB * 32);
        }
      }
      const float ia = pow2_field(254 - sa) * P.iD, ib = pow2_field(254 - sb) * P.iD;
      auto finish = [&](int j, const float (&l)[4]) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float s = r[j][v];
          if constexpr (C::SEP) s += e[j][v];
          r[j][v] = l[v] - s * (v < 2 ? ia : ib);
        }
      };
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        float4 a, b;
        if constexpr (C::SM) {
          a = load4<Np, V>(Qa, 16 * k + 4 * t), b = load4<Np, V>(Qb, 16 * k + 4 * t);
        } else {
          const float4 *d = reinterpret_cast<const float4 *>(sRp) + 2 * k * 32 + lane;
          a = d[0], b = d[32];
        }
        const float l0[4] = {a.x, a.y, b.x, b.y}, l1[4] = {a.z, a.w, b.z, b.w};
        finish(2 * k, l0);
        finish(2 * k + 1, l1);
      }
      if constexpr (KT) {
        float l[4];
        if constexpr (C::SM) {
          const float2 a = load2<Np, V>(Qa, 16 * KP + 2 * t), b = load2<Np, V>(Qb, 16 * KP + 2 * t);
          l[0] = a.x, l[1] = a.y, l[2] = b.x, l[3] = b.y;
        } else {
          const float4 a = reinterpret_cast<const float4 *>(sRp)[2 * KP * 32 + lane];
          l[0] = a.x, l[1] = a.y, l[2] = a.z, l[3] = a.w;
        }
        finish(2 * KP, l);
      }
    }
    if constexpr (C::SM) {  // the tile is consumed: the next one on its way
      __syncwarp();
      if (it + step < P.nit) fetch_tile(it + step);
    }

    // residual and old state of p, read while the projection runs
    constexpr bool PRE = NB <= 8;
    const float *pa = Qs + ea, *pb = Qs + eb;
    float4 pra[KP > 0 ? KP : 1], prb[KP > 0 ? KP : 1], pqa[KP > 0 ? KP : 1], pqb[KP > 0 ? KP : 1];
    if constexpr (PRE) {
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const int n = 16 * k + 4 * t;
        pra[k] = load4<Np, V>(Ra, n), prb[k] = load4<Np, V>(Rb, n);
        pqa[k] = load4<Np, V>(pa, n), pqb[k] = load4<Np, V>(pb, n);
      }
    }

    // ---- 4. WADG projection of rhs_p: 16 cubature points at a time through
    //         Vq, c2 and Pq
    float o[NB][4], oe[C::SEP ? NB : 1][4];
    float oia, oib;
    {
      Frag fr[KP > 0 ? KP : 1];
      Frag8 fr8;
      float ma = 0.f, mb = 0.f;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        ma = fmaxf(ma, fmaxf(fabsf(r[j][0]), fabsf(r[j][1])));
        mb = fmaxf(mb, fmaxf(fabsf(r[j][2]), fabsf(r[j][3])));
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          o[j][v] = 0.f;
          if constexpr (C::SEP) oe[j][v] = 0.f;
        }
      }
      ma = quad_max(ma), mb = quad_max(mb);
      const int sa = scale_field(ma), sb = scale_field(mb);
      const float ca = pow2_field(sa), cb = pow2_field(sb);
#pragma unroll
      for (int k = 0; k < KP; ++k)
        split_frag(fr[k], make_float4(r[2 * k][0], r[2 * k][1], r[2 * k + 1][0], r[2 * k + 1][1]),
                   make_float4(r[2 * k][2], r[2 * k][3], r[2 * k + 1][2], r[2 * k + 1][3]), ca, cb);
      if constexpr (KT)
        split_frag(fr8, make_float2(r[2 * KP][0], r[2 * KP][1]),
                   make_float2(r[2 * KP][2], r[2 * KP][3]), ca, cb);
      const float via = pow2_field(254 - sa) * P.iV, vib = pow2_field(254 - sb) * P.iV;
      // |Vq r| c2 <= vnorm max|r| max c2 bounds the weighted cubature values
      const int wa = scale_field(P.vnorm * ma * __ldg(P.c2max + ka)),
                wb = scale_field(P.vnorm * mb * __ldg(P.c2max + kb));
      const float da = pow2_field(wa), db = pow2_field(wb);
      oia = pow2_field(254 - wa) * P.iP, oib = pow2_field(254 - wb) * P.iP;
      const float4 *Ca = reinterpret_cast<const float4 *>(P.c2p + (size_t)ka * P.Nq16) + t,
                   *Cb = reinterpret_cast<const float4 *>(P.c2p + (size_t)kb * P.Nq16) + t;
      const int nch = P.Nq16 / 16;
      float4 za = __ldg(Ca), zb = __ldg(Cb);  // c2 at this chunk's points
#pragma unroll 1
      for (int c = 0; c < nch; ++c) {
        float v[4][4] = {};
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          const uint4 b0 = oV[((c * KP + k) * 2) * 32], b1 = oV[((c * KP + k) * 2 + 1) * 32];
          mma16(v[0], fr[k].h, b0.x, b0.y);
          mma16(v[1], fr[k].h, b1.x, b1.y);
          mma16(v[2], fr[k].h, b0.z, b0.w);
          mma16(v[3], fr[k].h, b1.z, b1.w);
          mma16(v[2], fr[k].l, b0.x, b0.y);
          mma16(v[3], fr[k].l, b1.x, b1.y);
          if constexpr (PR == 4) {
            mma16(v[2], fr[k].l, b0.z, b0.w);
            mma16(v[3], fr[k].l, b1.z, b1.w);
          }
        }
        if constexpr (KT) {
          const uint2 b0 = oVt[(c * 2) * 32], b1 = oVt[(c * 2 + 1) * 32];
          mma8(v[0], fr8.h[0], fr8.h[1], b0.x);
          mma8(v[1], fr8.h[0], fr8.h[1], b1.x);
          mma8(v[2], fr8.h[0], fr8.h[1], b0.y);
          mma8(v[3], fr8.h[0], fr8.h[1], b1.y);
          mma8(v[2], fr8.l[0], fr8.l[1], b0.x);
          mma8(v[3], fr8.l[0], fr8.l[1], b1.x);
          if constexpr (PR == 4) {
            mma8(v[2], fr8.l[0], fr8.l[1], b0.y);
            mma8(v[3], fr8.l[0], fr8.l[1], b1.y);
          }
        }
        // points 16 c + 4 t + 0 .. 3 of the two rows
        float4 xa = make_float4((v[0][0] + v[2][0]) * via, (v[0][1] + v[2][1]) * via,
                                (v[1][0] + v[3][0]) * via, (v[1][1] + v[3][1]) * via);
        float4 xb = make_float4((v[0][2] + v[2][2]) * vib, (v[0][3] + v[2][3]) * vib,
                                (v[1][2] + v[3][2]) * vib, (v[1][3] + v[3][3]) * vib);
        Frag w;
        xa = make_float4(xa.x * za.x, xa.y * za.y, xa.z * za.z, xa.w * za.w);
        xb = make_float4(xb.x * zb.x, xb.y * zb.y, xb.z * zb.z, xb.w * zb.w);
        split_frag(w, xa, xb, da, db);
        if (c + 1 < nch) za = __ldg(Ca + (c + 1) * 4), zb = __ldg(Cb + (c + 1) * 4);
        const uint4 *B = oP + c * NB * 32;
#pragma unroll
        for (int j0 = 0; j0 < NB; j0 += 4) {
          constexpr int full = NB / 4 * 4, rem = NB % 4 ? NB % 4 : 4;
          if (j0 < full) {
            uint4 b[4];
            float(&oo)[4][4] = *reinterpret_cast<float(*)[4][4]>(&o[j0]);
            float(&ee)[4][4] = *reinterpret_cast<float(*)[4][4]>(C::SEP ? &oe[C::SEP ? j0 : 0] : &o[j0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(oo, ee, w, b);
          } else {
            uint4 b[rem];
            float(&oo)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(&o[j0]);
            float(&ee)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(C::SEP ? &oe[C::SEP ? j0 : 0] : &o[j0]);
#pragma unroll
            for (int j = 0; j < rem; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(oo, ee, w, b);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if constexpr (C::SEP) o[j][v] += oe[j][v];
        o[j][v] *= v < 2 ? oia : oib;
      }

    // ---- 5. sources, added to the projected rhs_p
    //         (acous_elas_cpp/okl/ElasKernelsWADG.okl:400-403)
    if (P.src_tile) {
      const int tb = shot * P.nt32 + k0 / 32, te = shot * P.nt32 + min(k0 + 15, P.K - 1) / 32;
      const int j0 = __ldg(P.src_tile + tb), j1 = __ldg(P.src_tile + te + 1);
      if (j1 > j0) {
        const float amp = warp_ricker((float)(*P.time) + P.cstage * P.fdt, P.f0, P.tR, P.samp);
        for (int s = j0; s < j1; ++s) {
          const int e = __ldg(P.src_elem + s);
          if (e < k0 || e > k0 + 15) continue;
          const float *vec = P.src_vec + (size_t)s * Np;
          const bool xa = e == k0 + g, xb = e == k0 + g + 8;
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const int n = j < 2 * KP ? 16 * (j / 2) + 4 * t + 2 * (j & 1) : 16 * KP + 2 * t;
            const float s0 = n < Np ? amp * __ldg(vec + n) : 0.f;
            const float s1 = n + 1 < Np ? amp * __ldg(vec + n + 1) : 0.f;
            if (xa) o[j][0] += s0, o[j][1] += s1;
            if (xb) o[j][2] += s0, o[j][3] += s1;
          }
        }
      }
    }

    // ---- 6. LSRK update of p: res = fa res + fdt rhs, Q += fb res
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int n = 16 * k + 4 * t;
      if constexpr (!PRE) {
        pra[k] = load4<Np, V>(Ra, n), prb[k] = load4<Np, V>(Rb, n);
        pqa[k] = load4<Np, V>(pa, n), pqb[k] = load4<Np, V>(pb, n);
      }
      const float *x = o[2 * k], *y = o[2 * k + 1];
      float4 r, q;
      lsrk4(pra[k], make_float4(x[0], x[1], y[0], y[1]), pqa[k], P, r, q);
      if (va) {
        store4<Np, V>(Ra, n, r);
        store4<Np, V>(Oa, n, q);
      }
      lsrk4(prb[k], make_float4(x[2], x[3], y[2], y[3]), pqb[k], P, r, q);
      if (vb) {
        store4<Np, V>(Rb, n, r);
        store4<Np, V>(Ob, n, q);
      }
    }
    if constexpr (KT) {
      const int n = 16 * KP + 2 * t;
      const float2 ra = load2<Np, V>(Ra, n), rb = load2<Np, V>(Rb, n);
      const float2 qa = load2<Np, V>(pa, n), qb = load2<Np, V>(pb, n);
      const float *x = o[2 * KP];
      const float2 r2 = make_float2(P.fa * ra.x + P.fdt * x[0], P.fa * ra.y + P.fdt * x[1]);
      const float2 s2 = make_float2(P.fa * rb.x + P.fdt * x[2], P.fa * rb.y + P.fdt * x[3]);
      if (va) {
        store2<Np, V>(Ra, n, r2);
        store2<Np, V>(Oa, n, make_float2(qa.x + P.fb * r2.x, qa.y + P.fb * r2.y));
      }
      if (vb) {
        store2<Np, V>(Rb, n, s2);
        store2<Np, V>(Ob, n, make_float2(qb.x + P.fb * s2.x, qb.y + P.fb * s2.y));
      }
    }
  }
}

// ---------------------------------------------------------------- host side
template <int N>
static size_t warp_smem(const WarpPlan &pl, bool ops) {
  using C = WarpCfg<N>;
  return (ops ? (size_t)pl.ops_n * 16 : 0) + (size_t)pl.table_ints * 4 + (size_t)C::W * C::SCR * 4;
}

template <int N>
static bbw_status warp_launch_n(const WarpPlan &pl, const float *Qin, float *Qout, float *res,
                                float fa, float fb, float fdt, float cstage, cudaStream_t st) {
  using C = WarpCfg<N>;
  WarpParams P{};
  P.K = pl.K, P.K0 = pl.K0, P.Kc = pl.Kc > 0 ? pl.Kc : pl.K, P.Nq = pl.Nq, P.bc = pl.bc;
  P.pat_off = pl.pat_off, P.table_ints = pl.table_ints, P.nt32 = (pl.K + 31) / 32;
  P.Nq16 = (pl.Nq + 15) / 16 * 16;
  P.oDt = pl.oDt, P.oL = pl.oL, P.oLt = pl.oLt, P.oV = pl.oV, P.oVt = pl.oVt, P.oP = pl.oP;
  P.ops_n = pl.ops_n;
  P.fa = fa, P.fb = fb, P.fdt = fdt, P.cstage = cstage;
  P.iD = pl.iD, P.iL = pl.iL, P.iV = pl.iV, P.iP = pl.iP, P.vnorm = pl.vnorm;
  P.Qin = Qin, P.Qout = Qout, P.res = res;
  P.geo = pl.geo, P.c2p = pl.c2p, P.c2max = pl.c2max, P.nbr = pl.nbr;
  P.tables = pl.tables, P.ops = pl.ops;
  P.src_tile = pl.src_tile, P.src_elem = pl.src_elem, P.src_vec = pl.src_vec;
  P.f0 = pl.f0, P.tR = pl.tR, P.samp = pl.samp, P.time = pl.time;
  const int nt = (P.Kc - P.K0 + 15) / 16;
  P.nit = nt * pl.S;
  const int ctas = pl.max_ctas > 0 && pl.max_ctas < pl.nsm ? pl.max_ctas : pl.nsm;
  int grid;
  if (P.nit <= ctas * C::W) {
    // at most one item per warp: spread the items over the SMs first
    grid = P.nit < ctas ? P.nit : ctas;
    P.bs = 1, P.ws = grid;
  } else {
    // a CTA's warps walk neighbouring tiles, whose traces they share in L1
    grid = ctas;
    P.bs = C::W, P.ws = 1;
  }
  const size_t sm = warp_smem<N>(pl, pl.ops_sm);
  if constexpr (C::SM) {
    if (pl.ops_sm) {
      if (pl.products == 4) k_warp_stage<N, 4, true><<<grid, C::T, sm, st>>>(P);
      else k_warp_stage<N, 3, true><<<grid, C::T, sm, st>>>(P);
      return check_launch("warp-matrix stage");
    }
  }
  if (pl.products == 4) k_warp_stage<N, 4, false><<<grid, C::T, sm, st>>>(P);
  else k_warp_stage<N, 3, false><<<grid, C::T, sm, st>>>(P);
  return check_launch("warp-matrix stage");
}

template <int N>
static bbw_status warp_prepare_n(WarpPlan &pl) {
  const int maxsm = device_smem_optin();
  pl.ops_sm = WarpCfg<N>::SM && warp_smem<N>(pl, true) <= (size_t)maxsm;
  if (warp_smem<N>(pl, pl.ops_sm) > (size_t)maxsm)
    return set_error(BBW_ERR_UNSUPPORTED, "warp-matrix stage: does not fit in shared memory");
  std::vector<const void *> fn = {(const void *)k_warp_stage<N, 3, false>,
                                  (const void *)k_warp_stage<N, 4, false>};
  if constexpr (WarpCfg<N>::SM) {
    fn.push_back((const void *)k_warp_stage<N, 3, true>);
    fn.push_back((const void *)k_warp_stage<N, 4, true>);
  }
  for (const void *f : fn) {
    const bbw_status s = ensure_smem_limit(f, maxsm, "warp-matrix stage attribute");
    if (s != BBW_OK) return s;
  }
  return BBW_OK;
}

#define BBW_WARP_STAGE_INSTANCE(n)                                                              \
  bbw_status warp_launch_##n(const WarpPlan &pl, const float *Qin, float *Qout, float *res,     \
                             float fa, float fb, float fdt, float cstage, cudaStream_t st) {    \
    return warp_launch_n<n>(pl, Qin, Qout, res, fa, fb, fdt, cstage, st);                       \
  }                                                                                             \
  bbw_status warp_prepare_##n(WarpPlan &pl) { return warp_prepare_n<n>(pl); }

}  // namespace bbw
