// rk_volume, rk_surface and rk_update_WADG on warp-level matrix instructions
// (warp_mma.cuh) for the kernel-level entry points.
//
// The entry points take the reference's arrays as they are, so each CTA splits
// the operators into shared memory first (a few microseconds; pairs and a rest,
// as warp_pack does), then its warps
// walk 16-element tiles.  The kernels with a thread per node (kernels_ref.cu)
// spend one operator load and one or more shared loads per FMA; they stay for
// small meshes (matrix_form, kernels_ref.cu), N = 1, 2 and 8, and pointers that are
// not 16-byte aligned.
#pragma once
#include <vector>

#include "ref_mma.h"
#include "warp_mma.cuh"

namespace bbw {

// power of two that brings the CTA-wide maximum of |A| (n values) into [2^14,
// 2^15), as an exponent field; sRed: one int of shared memory, zero on entry
__device__ __forceinline__ void block_max(int *sRed, const float *__restrict__ A, int n) {
  float m = 0.f;
  for (int i0 = threadIdx.x; i0 < n; i0 += 16 * blockDim.x) {  // sixteen loads in flight
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = i0 + j * blockDim.x;
      v[j] = i < n ? fabsf(__ldg(A + i)) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) m = fmaxf(m, v[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(sRed, __float_as_int(m));
}
__device__ __forceinline__ int operator_field(int red) { return scale_field(__int_as_float(red)); }

// split tiles of the column-major nr x nc operator A times s into word `off` of
// the words at `out` (the rests in the plane at `rest`): row blocks rb, column
// pairs (k16) or the odd last block (k8); order [k][block]
template <bool K16>
__device__ __forceinline__ void split_tiles(uint32_t *out, uint32_t *rest, int off,
                                            const float *__restrict__ A, int nr, int nc, int nrp,
                                            int ncp, int nblk, int k0, int nk, float s) {
  const int tiles = nblk * nk;
#pragma unroll 4
  for (int i = threadIdx.x; i < tiles * 32; i += blockDim.x) {
    const int tl = i >> 5, lane = i & 31;
    const int r = slot_index(nrp, tl % nblk, lane >> 2);
    split_tile<K16>(out + off, rest + off / 4, i, k0 + tl / nblk, 2 * (lane & 3), s, [&](int b, int slot) {
      const int col = slot_index(ncp, b, slot);
      return r < nr && col < nc ? __ldg(A + r + (size_t)col * nr) : 0.f;
    });
  }
}

// first tile of worker w of a CTA: at most one tile per worker spreads them over
// the SMs, more go to neighbouring workers of one SM
__device__ __forceinline__ int first_tile(int nt, int per_cta, int w) {
  return nt <= (int)gridDim.x * per_cta ? blockIdx.x + w * gridDim.x : blockIdx.x * per_cta + w;
}

template <int N>
struct RefCfg {
  static constexpr int Np = NP(N), Nfp = NFP(N), NF = 4 * NFP(N), EW = 4 * Np;
  static constexpr int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2, U = KP + KT;
  static constexpr int FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  static constexpr int V = Np % 4 == 0 ? 4 : Np % 2 == 0 ? 2 : 1;
  static constexpr int W = 8, T = 256;
  static constexpr int OPS_VOL = 3 * NB * (KP * 128 + KT * 64);       // words
  static constexpr int OPS_SURF = 4 * NB * (FP * 128 + FT * 64);
  static constexpr int FLUX = 8 * FB * 8;
  // update: GW warps per tile, at most one unit of nodes each
  static constexpr int GW = U <= 2 ? U : U <= 4 ? 4 : 8, NG = (U <= 4 ? 12 : 8) / GW;
  static constexpr int TU = 32 * GW * NG;
  static constexpr int AS = KP * 64 + KT * 32;
  static constexpr int RC = N <= 3 ? 2 : 8;  // cubature chunks per round
  static constexpr int UPD = 16 * AS + RC * 4 * 256 + GW * 64 + RC * 64;  // floats per group
  static size_t ops_upd(int Nq) {  // words
    const size_t nch = (Nq + 15) / 16;
    return nch * (2 * (KP * 128 + KT * 64) + NB * 128);
  }
};

// ---------------------------------------------------------------- rk_volume
// cpp/okl/WaveKernels.okl:44-153
template <int N>
__global__ void __launch_bounds__(256, 1)
    k_rk_volume_mma(int K, const float *__restrict__ vgeo, const float *__restrict__ Dr,
                    const float *__restrict__ Ds, const float *__restrict__ Dt,
                    const float *__restrict__ Q, float *__restrict__ rhsQ) {
  using C = RefCfg<N>;
  constexpr int Np = C::Np, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW, V = C::V, PR = 4, PD = 5;
  extern __shared__ __align__(16) uint32_t smem_w[];
  uint32_t *rest = smem_w + C::OPS_VOL;
  int *sRed = reinterpret_cast<int *>(rest + C::OPS_VOL / 4);
  const int nt = (K + 15) / 16;
  if (threadIdx.x == 0) *sRed = 0;
  __syncthreads();
  block_max(sRed, Dr, Np * Np), block_max(sRed, Ds, Np * Np), block_max(sRed, Dt, Np * Np);
  __syncthreads();
  const int of = operator_field(*sRed);
  const float *D[3] = {Dr, Ds, Dt};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    split_tiles<true>(smem_w, rest, c * KP * NB * 128, D[c], Np, Np, Np, Np, NB, 0, KP, pow2_field(of));
    if constexpr (KT)
      split_tiles<false>(smem_w, rest, 3 * KP * NB * 128 + c * NB * 64, D[c], Np, Np, Np, Np, NB, 2 * KP,
                         1, pow2_field(of));
  }
  __syncthreads();
  const float iD = pow2_field(254 - of);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const uint4 *ops = reinterpret_cast<const uint4 *>(smem_w);
  const Ops<uint4, PR, false> oD(ops, rest, 0, lane);
  const Ops<uint2, PR, false> oDt(ops, rest, 3 * KP * NB * 32, lane);
  for (int it = first_tile(nt, C::W, warp); it < nt; it += gridDim.x * C::W) {
    const int ka = min(it * 16 + g, K - 1), kb = min(it * 16 + g + 8, K - 1);
    const bool va = it * 16 + g < K, vb = it * 16 + g + 8 < K;
    const float *Qa = Q + (size_t)ka * EW, *Qb = Q + (size_t)kb * EW;
    float *Ra = rhsQ + (size_t)ka * EW, *Rb = rhsQ + (size_t)kb * EW;
    float Ga[9], Gb[9];
#pragma unroll
    for (int c = 0; c < 9; ++c)
      Ga[c] = __ldg(vgeo + (size_t)ka * 9 + c), Gb[c] = __ldg(vgeo + (size_t)kb * 9 + c);
    {  // gradient of p
      Frag fp[KP > 0 ? KP : 1];
      Frag8 fp8;
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
      const float ia = -pow2_field(254 - sa) * iD, ib = -pow2_field(254 - sb) * iD;
#pragma unroll
      for (int k = 0; k < KP; ++k) split_frag(fp[k], xa[k], xb[k], pow2_field(sa), pow2_field(sb));
      if constexpr (KT) split_frag(fp8, ya, yb, pow2_field(sa), pow2_field(sb));
      // rhs of u, v, w at block j
      auto block = [&](int j, float (&rv)[3][4]) {
        float d[3][4] = {};
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          OpTile<uint4> b[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) b[c] = oD[((c * KP + k) * NB + j) * 32];
          mma_tiles<PD>(d, fp[k], b, N == 3 && k == 0);
        }
        if constexpr (KT) {
          OpTile<uint2> b[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) b[c] = oDt[(c * NB + j) * 32];
          mma_tiles<PD>(d, fp8, b);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const float *G = v < 2 ? Ga : Gb;
          const float s = v < 2 ? ia : ib;
          const float a = d[0][v] * s, b = d[1][v] * s, c = d[2][v] * s;
#pragma unroll
          for (int x = 0; x < 3; ++x) rv[x][v] = G[x] * a + G[3 + x] * b + G[6 + x] * c;
        }
      };
#pragma unroll 1
      for (int k = 0; k < KP; ++k) {
        float x[3][4], y[3][4];
        block(2 * k, x);
        block(2 * k + 1, y);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int n = 16 * k + 4 * t;
          if (va) store4<Np, V>(Ra + (c + 1) * Np, n, make_float4(x[c][0], x[c][1], y[c][0], y[c][1]));
          if (vb) store4<Np, V>(Rb + (c + 1) * Np, n, make_float4(x[c][2], x[c][3], y[c][2], y[c][3]));
        }
      }
      if constexpr (KT) {
        float x[3][4];
        block(2 * KP, x);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int n = 16 * KP + 2 * t;
          if (va) store2<Np, V>(Ra + (c + 1) * Np, n, make_float2(x[c][0], x[c][1]));
          if (vb) store2<Np, V>(Rb + (c + 1) * Np, n, make_float2(x[c][2], x[c][3]));
        }
      }
    }
    {  // divergence of the contravariant velocities
      float m[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          m[c] = max4(m[c], load4<Np, V>(Qa + (c + 1) * Np, 16 * k + 4 * t));
          m[3 + c] = max4(m[3 + c], load4<Np, V>(Qb + (c + 1) * Np, 16 * k + 4 * t));
        }
        if constexpr (KT) {
          m[c] = max2(m[c], load2<Np, V>(Qa + (c + 1) * Np, 16 * KP + 2 * t));
          m[3 + c] = max2(m[3 + c], load2<Np, V>(Qb + (c + 1) * Np, 16 * KP + 2 * t));
        }
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) m[c] = quad_max(m[c]);
      float Ma = 0.f, Mb = 0.f;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Ma = fmaxf(Ma, fabsf(Ga[3 * c]) * m[0] + fabsf(Ga[3 * c + 1]) * m[1] + fabsf(Ga[3 * c + 2]) * m[2]);
        Mb = fmaxf(Mb, fabsf(Gb[3 * c]) * m[3] + fabsf(Gb[3 * c + 1]) * m[4] + fabsf(Gb[3 * c + 2]) * m[5]);
      }
      const int sa = scale_field(2.f * Ma), sb = scale_field(2.f * Mb);
      const float ca = pow2_field(sa), cb = pow2_field(sb);
      float r[NB][4];
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) r[j][v] = 0.f;
      auto accumulate = [&](const auto &u, const auto B) {
        using T = decltype(B[0]);
        constexpr int full = NB / 4 * 4, rem = NB % 4;
#pragma unroll
        for (int j0 = 0; j0 < full; j0 += 4) {
          T b[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) b[j] = B[(j0 + j) * 32];
          mma_tiles<PD>(*reinterpret_cast<float(*)[4][4]>(&r[j0]), u, b);
        }
        if constexpr (rem > 0) {
          T b[rem];
#pragma unroll
          for (int j = 0; j < rem; ++j) b[j] = B[(full + j) * 32];
          mma_tiles<PD>(*reinterpret_cast<float(*)[rem][4]>(&r[full]), u, b);
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
      const float ia = -pow2_field(254 - sa) * iD, ib = -pow2_field(254 - sb) * iD;
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) r[j][v] *= v < 2 ? ia : ib;
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const int n = 16 * k + 4 * t;
        const float *x = r[2 * k], *y = r[2 * k + 1];
        if (va) store4<Np, V>(Ra, n, make_float4(x[0], x[1], y[0], y[1]));
        if (vb) store4<Np, V>(Rb, n, make_float4(x[2], x[3], y[2], y[3]));
      }
      if constexpr (KT) {
        const int n = 16 * KP + 2 * t;
        if (va) store2<Np, V>(Ra, n, make_float2(r[2 * KP][0], r[2 * KP][1]));
        if (vb) store2<Np, V>(Rb, n, make_float2(r[2 * KP][2], r[2 * KP][3]));
      }
    }
  }
}

// --------------------------------------------------------------- rk_surface
// cpp/okl/WaveKernels.okl:156-260
// fluxes of face f at nodes I0 .. I0 + NI - 1 of eight elements k0 .. k0 + 7
template <int N, int I0, int NI>
__device__ __forceinline__ void ref_face_flux(int K, int bc, const float *__restrict__ fgeo,
                                              const int *__restrict__ Fmask,
                                              const int *__restrict__ vmapP,
                                              const float *__restrict__ Q, float *sF, int f, int k0,
                                              int lane) {
  using C = RefCfg<N>;
  constexpr int Np = C::Np, EPI = NI >= 32 ? 1 : (32 / NI > 8 ? 8 : 32 / NI), IT = (8 + EPI - 1) / EPI;
  const bool act = lane / NI < EPI;
  const int sub = act ? lane / NI : 0, i = I0 + (act ? lane % NI : 0);
  const int own = __ldg(Fmask + f * C::Nfp + i);
  const float wp = bc == BBW_BC_PRESSURE_RELEASE ? -1.f : 1.f, wu = -wp;
  int idP[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it)
    idP[it] = __ldg(vmapP + (size_t)min(k0 + min(it * EPI + sub, 7), K - 1) * C::NF + f * C::Nfp + i);
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = it * EPI + sub, k = min(k0 + min(e, 7), K - 1);
    const float *m = Q + (size_t)k * C::EW + own, *x = Q + idP[it];
    const bool wall = idP[it] == k * C::EW + own;
    const float *gp = fgeo + ((size_t)k * 4 + f) * 4;
    const float Fs = __ldg(gp), nx = __ldg(gp + 1), ny = __ldg(gp + 2), nz = __ldg(gp + 3);
    // a wall's + trace is the own one with p or the velocity reversed
    const float sp = wall ? wp : 1.f, su = wall ? wu : 1.f;
    const float dp = fmaf(sp, __ldg(x), -__ldg(m));
    float un = fmaf(su, __ldg(x + Np), -__ldg(m + Np)) * nx;
    un = fmaf(fmaf(su, __ldg(x + 2 * Np), -__ldg(m + 2 * Np)), ny, un);
    un = fmaf(fmaf(su, __ldg(x + 3 * Np), -__ldg(m + 3 * Np)), nz, un);
    if (act && e < 8) sF[e * (8 * C::FB) + i] = .5f * Fs * (dp - un);
  }
}

template <int N>
__global__ void __launch_bounds__(256, 1)
    k_rk_surface_mma(int K, int bc, const float *__restrict__ fgeo, const int *__restrict__ Fmask,
                     const int *__restrict__ vmapP, const float *__restrict__ LIFT,
                     const float *__restrict__ Q, float *__restrict__ rhsQ) {
  using C = RefCfg<N>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW, V = C::V;
  constexpr int FB = C::FB, FP = C::FP, FT = C::FT;
  extern __shared__ __align__(16) uint32_t smem_w[];
  uint32_t *rest = smem_w + C::OPS_SURF;
  int *sRed = reinterpret_cast<int *>(rest + C::OPS_SURF / 4);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  float *sF = reinterpret_cast<float *>(sRed + 4) + warp * C::FLUX;
  const int nt = (K + 15) / 16;
  if (threadIdx.x == 0) *sRed = 0;
  for (int i = lane; i < C::FLUX; i += 32) sF[i] = 0.f;  // columns past Nfp stay zero
  __syncthreads();
  block_max(sRed, LIFT, Np * 4 * Nfp);
  __syncthreads();
  const int of = operator_field(*sRed);
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const float *L = LIFT + (size_t)f * Nfp * Np;
    split_tiles<true>(smem_w, rest, f * FP * NB * 128, L, Np, Nfp, Np, Nfp, NB, 0, FP, pow2_field(of));
    if constexpr (FT)
      split_tiles<false>(smem_w, rest, 4 * FP * NB * 128 + f * NB * 64, L, Np, Nfp, Np, Nfp, NB, 2 * FP, 1,
                         pow2_field(of));
  }
  __syncthreads();
  const float iL = pow2_field(254 - of);
  const uint4 *ops = reinterpret_cast<const uint4 *>(smem_w);
  const Ops<uint4, 4, false> oL(ops, rest, 0, lane);
  const Ops<uint2, 4, false> oLt(ops, rest, 4 * FP * NB * 32, lane);
  for (int it = first_tile(nt, C::W, warp); it < nt; it += gridDim.x * C::W) {
    const int k0 = it * 16, ka = min(k0 + g, K - 1), kb = min(k0 + g + 8, K - 1);
    const bool va = k0 + g < K, vb = k0 + g + 8 < K;
    float *Ra = rhsQ + (size_t)ka * EW, *Rb = rhsQ + (size_t)kb * EW;
    Frag ff[4][FP > 0 ? FP : 1];
    Frag8 f8[4];
    float na[4][4], nb[4][4];  // inverse flux scale, and minus it times the normal
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      float inv[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        __syncwarp();
        if constexpr (Nfp <= 32) {
          ref_face_flux<N, 0, Nfp>(K, bc, fgeo, Fmask, vmapP, Q, sF, f, k0 + 8 * h, lane);
        } else {
          ref_face_flux<N, 0, 32>(K, bc, fgeo, Fmask, vmapP, Q, sF, f, k0 + 8 * h, lane);
          ref_face_flux<N, 32, Nfp - 32>(K, bc, fgeo, Fmask, vmapP, Q, sF, f, k0 + 8 * h, lane);
        }
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
        const float2 cs = both(pow2_field(sc));
        inv[h] = pow2_field(254 - sc) * iL;
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          split2(lo2(x[k]), cs, ff[f][k].h[h], ff[f][k].l[h]);
          split2(hi2(x[k]), cs, ff[f][k].h[2 + h], ff[f][k].l[2 + h]);
        }
        if constexpr (FT) split2(y, cs, f8[f].h[h], f8[f].l[h]);
      }
      const float *pa = fgeo + ((size_t)ka * 4 + f) * 4, *pb = fgeo + ((size_t)kb * 4 + f) * 4;
      na[f][0] = inv[0], nb[f][0] = inv[1];
#pragma unroll
      for (int x = 1; x < 4; ++x) na[f][x] = -__ldg(pa + x) * inv[0], nb[f][x] = -__ldg(pb + x) * inv[1];
    }
    // lifted fluxes of block j: four fields
    auto block = [&](int j, float (&r)[4][4]) {
      float L[4][4] = {};
      auto step = [&](const auto &x, const auto (&b)[4]) {
        float t4[4][4];
#pragma unroll
        for (int p = 0; p < kProducts; ++p)
#pragma unroll
          for (int f = 0; f < 4; ++f) mma_step<4>(t4[f], x(f), b[f], p);
#pragma unroll
        for (int f = 0; f < 4; ++f) add4(L[f], t4[f]);
      };
#pragma unroll
      for (int k = 0; k < FP; ++k) {
        OpTile<uint4> b[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) b[f] = oL[((f * FP + k) * NB + j) * 32];
        step([&](int f) { return ff[f][k]; }, b);
      }
      if constexpr (FT) {
        OpTile<uint2> b[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) b[f] = oLt[(f * NB + j) * 32];
        step([&](int f) { return f8[f]; }, b);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float s = 0.f;
#pragma unroll
          for (int f = 0; f < 4; ++f) s = fmaf(L[f][v], v < 2 ? na[f][x] : nb[f][x], s);
          r[x][v] = s;
        }
    };
#pragma unroll 1
    for (int k = 0; k < KP; ++k) {
      const int n = 16 * k + 4 * t;
      float4 oa[4], ob[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) oa[c] = load4<Np, V>(Ra + c * Np, n), ob[c] = load4<Np, V>(Rb + c * Np, n);
      float x[4][4], y[4][4];
      block(2 * k, x);
      block(2 * k + 1, y);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (va)
          store4<Np, V>(Ra + c * Np, n, make_float4(oa[c].x + x[c][0], oa[c].y + x[c][1],
                                                    oa[c].z + y[c][0], oa[c].w + y[c][1]));
        if (vb)
          store4<Np, V>(Rb + c * Np, n, make_float4(ob[c].x + x[c][2], ob[c].y + x[c][3],
                                                    ob[c].z + y[c][2], ob[c].w + y[c][3]));
      }
    }
    if constexpr (KT) {
      const int n = 16 * KP + 2 * t;
      float2 oa[4], ob[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) oa[c] = load2<Np, V>(Ra + c * Np, n), ob[c] = load2<Np, V>(Rb + c * Np, n);
      float x[4][4];
      block(2 * KP, x);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (va) store2<Np, V>(Ra + c * Np, n, make_float2(oa[c].x + x[c][0], oa[c].y + x[c][1]));
        if (vb) store2<Np, V>(Rb + c * Np, n, make_float2(ob[c].x + x[c][2], ob[c].y + x[c][3]));
      }
    }
  }
}

// ----------------------------------------------------------- rk_update_WADG
// cpp/okl/WaveKernelsWADG.okl:1760-1887
template <int N>
__global__ void __launch_bounds__(RefCfg<N>::TU, 1)
    k_rk_update_mma(int K, int Nq, const float *__restrict__ Vq, const float *__restrict__ Pq,
                    const float *__restrict__ Jq, const float *__restrict__ c2q, float fa, float fb,
                    float fdt, const float *__restrict__ rhsQ, float *__restrict__ resQ,
                    float *__restrict__ Q) {
  using C = RefCfg<N>;
  constexpr int Np = C::Np, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW, V = C::V, GW = C::GW;
  constexpr int AS = C::AS, RC = C::RC, PR = 4;
  extern __shared__ __align__(16) uint32_t smem_w[];
  const int nch = (Nq + 15) / 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int grp = warp / GW, w = warp - grp * GW;
  // operators: Vq [chunk][KP][2], its k8 tails [chunk][2], Pq [chunk][NB]
  const int aVt = nch * KP * 2 * 128, aP = aVt + nch * KT * 2 * 64, aM = aP + nch * NB * 128;  // words
  uint32_t *rest = smem_w + aM;
  int *sRed = reinterpret_cast<int *>(rest + aM / 4);
  float *scr = reinterpret_cast<float *>(sRed + 4) + grp * C::UPD;
  const int nt = (K + 15) / 16;
  if (threadIdx.x < 2) sRed[threadIdx.x] = 0;
  __syncthreads();
  block_max(sRed, Vq, Nq * Np), block_max(sRed + 1, Pq, Nq * Np);
  __syncthreads();
  const int ov = operator_field(sRed[0]), op = operator_field(sRed[1]);
  // row block 2 chunk + h, steps k: tile (chunk, k, h)
#pragma unroll 4
  for (int i = threadIdx.x; i < nch * 2 * KP * 32; i += blockDim.x) {
    const int tl = i >> 5, l = i & 31, h = tl & 1, k = (tl >> 1) % (KP > 0 ? KP : 1), c = (tl >> 1) / (KP > 0 ? KP : 1);
    const int r = slot_index(16 * nch, 2 * c + h, l >> 2);
    split_tile<true>(smem_w, rest, i, k, 2 * (l & 3), pow2_field(ov), [&](int b, int slot) {
      const int col = slot_index(Np, b, slot);
      return r < Nq && col < Np ? __ldg(Vq + r + (size_t)col * Nq) : 0.f;
    });
  }
  if constexpr (KT)
    split_tiles<false>(smem_w, rest, aVt, Vq, Nq, Np, 16 * nch, Np, 2 * nch, 2 * KP, 1, pow2_field(ov));
  split_tiles<true>(smem_w, rest, aP, Pq, Np, Nq, Np, 16 * nch, NB, 0, nch, pow2_field(op));
  __syncthreads();
  const float iV = pow2_field(254 - ov), iP = pow2_field(254 - op);
  const uint4 *ops = reinterpret_cast<const uint4 *>(smem_w);
  const Ops<uint4, PR, false> oV(ops, rest, 0, lane), oP(ops, rest, aP / 4, lane);
  const Ops<uint2, PR, false> oVt(ops, rest, aVt / 4, lane);
  uint4 *sA = reinterpret_cast<uint4 *>(scr);                 // split rhs, four fields
  uint4 *sW = reinterpret_cast<uint4 *>(scr + 16 * AS);       // split point values [RC][4]
  float4 *sMax = reinterpret_cast<float4 *>(scr + 16 * AS + RC * 1024);  // [GW][16]
  float4 *sInv = sMax + GW * 16;                              // [RC][16] inverse scales
  const bool mine = w < C::U, pair = w < KP;
  for (int it = first_tile(nt, C::NG, grp); it < nt; it += gridDim.x * C::NG) {
    const int ka = min(it * 16 + g, K - 1), kb = min(it * 16 + g + 8, K - 1);
    const bool va = it * 16 + g < K, vb = it * 16 + g + 8 < K;
    const size_t ea = (size_t)ka * EW, eb = (size_t)kb * EW;
    float4 xa[4], xb[4];
    float m[8];
    auto unit = [&](const float *p, int c) {
      if (!mine) return make_float4(0.f, 0.f, 0.f, 0.f);
      if (pair) return load4<Np, V>(p + c * Np, 16 * w + 4 * t);
      const float2 y = load2<Np, V>(p + c * Np, 16 * KP + 2 * t);
      return make_float4(y.x, y.y, 0.f, 0.f);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      xa[c] = unit(rhsQ + ea, c), xb[c] = unit(rhsQ + eb, c);
      m[c] = quad_max(max4(0.f, xa[c])), m[4 + c] = quad_max(max4(0.f, xb[c]));
    }
    if (t < 2)
      sMax[w * 16 + g + 8 * t] = t == 0 ? make_float4(m[0], m[1], m[2], m[3]) : make_float4(m[4], m[5], m[6], m[7]);
    group_sync<GW>(grp);  // maxima ready; the previous tile is consumed
    float4 ma = sMax[g], mb = sMax[g + 8];
#pragma unroll
    for (int i = 1; i < GW; ++i) {
      const float4 a = sMax[i * 16 + g], b = sMax[i * 16 + g + 8];
      ma = make_float4(fmaxf(ma.x, a.x), fmaxf(ma.y, a.y), fmaxf(ma.z, a.z), fmaxf(ma.w, a.w));
      mb = make_float4(fmaxf(mb.x, b.x), fmaxf(mb.y, b.y), fmaxf(mb.z, b.z), fmaxf(mb.w, b.w));
    }
    const int sf[4][2] = {{scale_field(ma.x), scale_field(mb.x)}, {scale_field(ma.y), scale_field(mb.y)},
                          {scale_field(ma.z), scale_field(mb.z)}, {scale_field(ma.w), scale_field(mb.w)}};
    if (mine) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (pair) {
          Frag f;
          split_frag(f, xa[c], xb[c], pow2_field(sf[c][0]), pow2_field(sf[c][1]));
          put_frag(sA + c * AS, w, lane, f);
        } else {
          Frag8 f;
          split_frag(f, lo2(xa[c]), lo2(xb[c]), pow2_field(sf[c][0]), pow2_field(sf[c][1]));
          put_frag8(sA + c * AS, KP, lane, f);
        }
      }
    }
    group_sync<GW>(grp);
    float r[4][2][4] = {};
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += RC) {
      const int cend = min(nch, c0 + RC);
      if (c0 > 0) group_sync<GW>(grp);
#pragma unroll 1
      for (int c = c0 + w; c < cend; c += GW) {
        // weights 1/J and c2 at points 16 c + 4 t + 0 .. 3 of rows a and b
        float wj[2][4], wc[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = 16 * c + 4 * t + q;
            const size_t at = (size_t)(h ? kb : ka) * Nq + (i < Nq ? i : 0);
            wj[h][q] = i < Nq ? 1.f / __ldg(Jq + at) : 0.f;
            wc[h][q] = i < Nq ? __ldg(c2q + at) : 0.f;
          }
        float v[4][2][4] = {};
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          const OpTile<uint4> b[2] = {oV[((c * KP + k) * 2) * 32], oV[((c * KP + k) * 2 + 1) * 32]};
#pragma unroll
          for (int x = 0; x < 4; x += 2)
            mma_pair2<PR, PR>(v[x], get_frag(sA + x * AS, k, lane), b, v[x + 1],
                          get_frag(sA + (x + 1) * AS, k, lane), b);
        }
        if constexpr (KT) {
          const OpTile<uint2> b[2] = {oVt[(c * 2) * 32], oVt[(c * 2 + 1) * 32]};
#pragma unroll
          for (int x = 0; x < 4; x += 2)
            mma_pair2<PR, PR>(v[x], get_frag8(sA + x * AS, KP, lane), b, v[x + 1],
                          get_frag8(sA + (x + 1) * AS, KP, lane), b);
        }
        float4 inva, invb;
        float *ia = &inva.x, *ib = &invb.x;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float y[2][4], mm[2] = {0.f, 0.f};
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = q / 2, j = 2 * h + q % 2;
              float z = v[x][i][j] * (pow2_field(254 - sf[x][h]) * iV) * wj[h][q];
              if (x == 0) z *= wc[h][q];
              y[h][q] = z;
              mm[h] = fmaxf(mm[h], fabsf(z));
            }
          const int fa_ = scale_field(quad_max(mm[0])), fb_ = scale_field(quad_max(mm[1]));
          ia[x] = pow2_field(254 - fa_) * iP, ib[x] = pow2_field(254 - fb_) * iP;
          Frag f;
          split_frag(f, make_float4(y[0][0], y[0][1], y[0][2], y[0][3]),
                     make_float4(y[1][0], y[1][1], y[1][2], y[1][3]), pow2_field(fa_), pow2_field(fb_));
          put_frag(sW + ((c - c0) * 4 + x) * 64, 0, lane, f);
        }
        if (t == 0) sInv[(c - c0) * 16 + g] = inva, sInv[(c - c0) * 16 + g + 8] = invb;
      }
      group_sync<GW>(grp);
#pragma unroll 1
      for (int c = c0; c < cend && mine; ++c) {
        const uint4 *W = sW + (c - c0) * 4 * 64;
        const OpTile<uint4> b[2] = {oP[(c * NB + 2 * w) * 32], oP[(c * NB + 2 * w + (pair ? 1 : 0)) * 32]};
        const float4 va4 = sInv[(c - c0) * 16 + g], vb4 = sInv[(c - c0) * 16 + g + 8];
        const float ia[4] = {va4.x, va4.y, va4.z, va4.w}, ib[4] = {vb4.x, vb4.y, vb4.z, vb4.w};
        float o[4][2][4] = {};
#pragma unroll
        for (int x = 0; x < 4; x += 2)
          mma_pair2<PR, PR>(o[x], get_frag(W + x * 64, 0, lane), b, o[x + 1],
                        get_frag(W + (x + 1) * 64, 0, lane), b);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              r[x][i][j] = fmaf(o[x][i][j], j < 2 ? ia[x] : ib[x], r[x][i][j]);
      }
    }
    const float2 fa2 = both(fa), fd2 = both(fdt), fb2 = both(fb);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!mine || !(h ? vb : va)) continue;
        const size_t at = (h ? eb : ea) + c * Np;
        const float2 x0 = make_float2(r[c][0][2 * h], r[c][0][2 * h + 1]);
        if (pair) {
          const float2 x1 = make_float2(r[c][1][2 * h], r[c][1][2 * h + 1]);
          const int n = 16 * w + 4 * t;
          const float4 old = load4<Np, V>(resQ + at, n), q = load4<Np, V>(Q + at, n);
          const float2 y0 = lsrk2(lo2(old), x0, fa2, fd2), y1 = lsrk2(hi2(old), x1, fa2, fd2);
          const float2 z0 = __ffma2_rn(fb2, y0, lo2(q)), z1 = __ffma2_rn(fb2, y1, hi2(q));
          store4<Np, V>(resQ + at, n, make_float4(y0.x, y0.y, y1.x, y1.y));
          store4<Np, V>(Q + at, n, make_float4(z0.x, z0.y, z1.x, z1.y));
        } else {
          const int n = 16 * KP + 2 * t;
          const float2 y = lsrk2(load2<Np, V>(resQ + at, n), x0, fa2, fd2);
          const float2 z = __ffma2_rn(fb2, y, load2<Np, V>(Q + at, n));
          store2<Np, V>(resQ + at, n, y);
          store2<Np, V>(Q + at, n, z);
        }
      }
  }
}

// ---------------------------------------------------------------- host side
inline int ref_grid(int K) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (nsm <= 0) nsm = 148;
  const int need = (K + 15) / 16;
  return need < nsm ? need : nsm;
}

template <int N>
static bbw_status ref_volume_n(int K, const float *vgeo, const float *Dr, const float *Ds,
                               const float *Dt, const float *Q, float *rhsQ, cudaStream_t st) {
  using C = RefCfg<N>;
  const int sm = C::OPS_VOL * 5 + 16;
  const bbw_status s = ensure_smem_limit(k_rk_volume_mma<N>, sm, "rk_volume attribute");
  if (s != BBW_OK) return s;
  k_rk_volume_mma<N><<<ref_grid(K), 256, sm, st>>>(K, vgeo, Dr, Ds, Dt, Q, rhsQ);
  return check_launch("rk_volume");
}

template <int N>
static bbw_status ref_surface_n(int K, int bc, const float *fgeo, const int *Fmask, const int *vmapP,
                                const float *LIFT, const float *Q, float *rhsQ, cudaStream_t st) {
  using C = RefCfg<N>;
  const int sm = C::OPS_SURF * 5 + 16 + C::W * C::FLUX * 4;
  const bbw_status s = ensure_smem_limit(k_rk_surface_mma<N>, sm, "rk_surface attribute");
  if (s != BBW_OK) return s;
  k_rk_surface_mma<N><<<ref_grid(K), 256, sm, st>>>(K, bc, fgeo, Fmask, vmapP, LIFT, Q, rhsQ);
  return check_launch("rk_surface");
}

template <int N>
static size_t ref_update_smem(int Nq) {
  using C = RefCfg<N>;
  return C::ops_upd(Nq) * 5 + 16 + (size_t)C::NG * C::UPD * 4;
}

template <int N>
static bbw_status ref_update_n(int K, int Nq, const float *Vq, const float *Pq, const float *Jq,
                               const float *c2q, float fa, float fb, float fdt, const float *rhsQ,
                               float *resQ, float *Q, cudaStream_t st) {
  using C = RefCfg<N>;
  const size_t sm = ref_update_smem<N>(Nq);
  const bbw_status s = ensure_smem_limit(k_rk_update_mma<N>, device_smem_optin(), "rk_update_WADG attribute");
  if (s != BBW_OK) return s;
  k_rk_update_mma<N><<<ref_grid(K), C::TU, sm, st>>>(K, Nq, Vq, Pq, Jq, c2q, fa, fb, fdt, rhsQ, resQ, Q);
  return check_launch("rk_update_WADG");
}

#define BBW_REF_RHS_INSTANCE(n)                                                                  \
  bbw_status ref_volume_##n(int K, const float *vgeo, const float *Dr, const float *Ds,          \
                            const float *Dt, const float *Q, float *rhsQ, cudaStream_t st) {     \
    return ref_volume_n<n>(K, vgeo, Dr, Ds, Dt, Q, rhsQ, st);                                    \
  }                                                                                              \
  bbw_status ref_surface_##n(int K, int bc, const float *fgeo, const int *Fmask, const int *vmapP, \
                             const float *LIFT, const float *Q, float *rhsQ, cudaStream_t st) {  \
    return ref_surface_n<n>(K, bc, fgeo, Fmask, vmapP, LIFT, Q, rhsQ, st);                       \
  }
#define BBW_REF_UPDATE_INSTANCE(n)                                                               \
  bool ref_update_fits_##n(int Nq) { return ref_update_smem<n>(Nq) <= (size_t)device_smem_optin(); } \
  bbw_status ref_update_##n(int K, int Nq, const float *Vq, const float *Pq, const float *Jq,    \
                            const float *c2q, float fa, float fb, float fdt, const float *rhsQ,  \
                            float *resQ, float *Q, cudaStream_t st) {                            \
    return ref_update_n<n>(K, Nq, Vq, Pq, Jq, c2q, fa, fb, fdt, rhsQ, resQ, Q, st);              \
  }

}  // namespace bbw
