// One LSRK stage with every contraction on warp-level matrix instructions
// (warp_mma.cuh), one warp per 16-element tile.
//
// Replaces rk_volume + rk_surface + rk_update_WADG of the reference
// (cpp/okl/WaveKernels.okl:44-260, cpp/okl/WaveKernelsWADG.okl:1760-1887).
//
// A warp owns its tile from the trace gather to the LSRK update: rhs_p -> Vq ->
// c2 -> Pq chains in registers, without shared memory or any barrier between
// warps.  Bound by instruction latency at two or three warps per scheduler
// (issue 27 %, HBM 34 %); us per stage, CTA-wide FP32 stage -> this form: N = 2,
// K = 93750: 94 -> 46; N = 3, K = 196608: 310 -> 137; N = 4, K = 82944: 249 -> 128.
#pragma once
#include <vector>

#include "warp_mma.cuh"

namespace bbw {

template <int N>
struct WarpCfg {
  static_assert(N <= 4, "one warp per tile: N <= 4");
  static constexpr int Np = NP(N), Nfp = NFP(N), EW = 4 * Np;
  // blocks of eight nodes: pairs of them are the k16 steps, an odd last one
  // is a k8 step (same for the face nodes)
  static constexpr int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2;
  static constexpr int FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  // warps per CTA: 255 registers at N = 3 and 4 (12 warps at 168 registers
  // spill: 143.6 against 141.3 us at N = 3, K = 196608)
  static constexpr int W = N <= 2 ? 12 : 8;
  static constexpr int T = 32 * W;
  static constexpr int V = Np % 4 == 0 ? 4 : Np % 2 == 0 ? 2 : 1;  // vector width of a row
  // state tile of a warp: rows of 4 Np floats, padded so that two rows of a
  // pair start 16 banks apart (a 16-byte access serves two rows at a time)
  static constexpr int ODD = V == 4 ? (48 - EW % 32) % 32 : 0;
  static constexpr int TILE = 16 * EW + 8 * ODD;
  __host__ __device__ static constexpr int row(int e) { return e * EW + ((e + 1) >> 1) * ODD; }
  static constexpr int FLUX = 8 * FB * 8;  // eight elements' fluxes
  static constexpr int SCR = TILE + FLUX;
};

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
                                       const int *sTab, int f, int h8, int k0, int code, int lane) {
    const int i = node(lane);
    const float4 *geo = reinterpret_cast<const float4 *>(P.geo) + (size_t)(k0 + h8) * 7 + f;
    walls = 0;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = elem(it, lane);
      const int cd = __shfl_sync(0xffffffffu, code, e * 4 + f);
      const int pat = cd & 255;
      const bool wall = pat == 255;
      walls |= wall ? 1u << it : 0u;
      // a wall's + trace is the own face node (the table starts with Fmask)
      const int nn = sTab[(wall ? f * C::Nfp : P.pat_off + pat * C::Nfp) + i];
      const float *x = Qs + (size_t)(cd >> 8) * C::EW + nn;
#pragma unroll
      for (int c = 0; c < 4; ++c) X[it][c] = __ldg(x + c * C::Np);
      g[it] = __ldg(geo + e * 7);
    }
  }
  // upwind pressure flux to sF[element][8 FB].  A wall's + trace is the own
  // one with the pressure (p = 0 wall) or the velocity (rigid) reversed.
  __device__ __forceinline__ void flux(const WarpParams &P, const float *sQ, const int *sFm,
                                       float *sF, int f, int h8, int lane) const {
    const bool act = lane / NI < EPI;
    const int i = node(lane), own = sFm[f * C::Nfp + i];
    const float wp = P.bc == BBW_BC_PRESSURE_RELEASE ? -1.f : 1.f, wu = -wp;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = elem(it, lane);
      const float *m = sQ + C::row(h8 + e) + own;
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
  // operators and tables, all copies in flight with the first tile's
  if constexpr (OPS) stage_async<C::T>(sOps, P.ops, P.ops_n);
  stage_async<C::T>(reinterpret_cast<uint4 *>(sTab), reinterpret_cast<const uint4 *>(P.tables),
                    P.table_ints / 4);
  float *sQ = scr, *sF = scr + C::TILE;
  if constexpr (FB * 8 > Nfp)  // flux columns past Nfp meet zero operator columns
    for (int i = lane; i < C::FLUX; i += 32) sF[i] = 0.f;
  const uint4 *ops = OPS ? sOps : P.ops;
  constexpr int PD = PR == 4 ? 5 : PR;  // derivatives: large terms cancel
  // a sum's first step sets it instead of adding to zero; by the registers it pays at
  // N = 3 only (us per stage added / set: N = 2, K = 93750 45.3 / 45.7, N = 3, K = 82944
  // 63.9 / 61.6, N = 4, K = 24576 48.5 / 49.1)
  constexpr bool SET = N == 3;
  using O16 = Ops<uint4, PR, !OPS>;
  using O8 = Ops<uint2, PR, !OPS>;
  const void *rests = ops + P.oM;
  const O16 oD(ops, rests, 0, lane), oL(ops, rests, P.oL, lane), oV(ops, rests, P.oV, lane),
      oP(ops, rests, P.oP, lane);
  const O8 oDt(ops, rests, P.oDt, lane), oLt(ops, rests, P.oLt, lane), oVt(ops, rests, P.oVt, lane);
  const int klast = P.Kc - 1;
  const size_t shot_stride = (size_t)P.K * EW;
  const int step = gridDim.x * C::W;

  // state tile of item i to shared memory; neighbour codes of its faces
  auto fetch_tile = [&](int sh, int kn) {
    const int ne = min(16, P.Kc - kn);
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
  auto codes = [&](int kn, int &c0, int &c1) {
    c0 = __ldg(P.nbr + (size_t)min(kn + g, klast) * 4 + t);
    c1 = __ldg(P.nbr + (size_t)min(kn + 8 + g, klast) * 4 + t);
  };

  int it = blockIdx.x * P.bs + warp * P.ws;
  int code0 = 0, code1 = 0;
  int nshot = it / P.ntile, ntl = it - nshot * P.ntile;  // the next item
  if (it < P.nit) {
    fetch_tile(nshot, P.K0 + ntl * 16);
    codes(P.K0 + ntl * 16, code0, code1);
  }
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
    float *Qa = sQ + C::row(ka - k0);
    float *Qb = sQ + C::row(kb - k0);
    float *Ra = P.res + shot * shot_stride + ea, *Rb = P.res + shot * shot_stride + eb;
    float *Oa = P.Qout + shot * shot_stride + ea, *Ob = P.Qout + shot * shot_stride + eb;

    if (lane == 0) {  // the next item's inputs on their way to L2
      if (it + step < P.nit) {
        const int ne = min(16, P.Kc - kn);
        const size_t at = nshot * shot_stride + (size_t)kn * EW;
        prefetch_l2(P.Qin + at, (size_t)ne * EW * 4);
        prefetch_l2(P.res + at, (size_t)ne * EW * 4);
        prefetch_l2(P.c2p + (size_t)kn * P.Nq16, (size_t)ne * P.Nq16 * 4);
      }
    }
    cp_async_wait();
    __syncwarp();

    // ---- 1. face fluxes of eight elements at a time (the rows l/4, then
    //         l/4 + 8); the next half face's gather is in flight meanwhile
    Frag ff[4][FP > 0 ? FP : 1];
    Frag8 f8[4];
    float fia[4], fib[4];  // inverse scales of the faces
    {
      FaceGather<N, 0, Nfp> buf[2];
      buf[0].load(P, Qs, sTab, 0, 0, k0, code0, lane);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int f = r >> 1, h = r & 1;
        if (r < 7)
          buf[(r + 1) & 1].load(P, Qs, sTab, (r + 1) >> 1, 8 * ((r + 1) & 1), k0,
                                (r + 1) & 1 ? code1 : code0, lane);
        buf[r & 1].flux(P, sQ, sTab, sF, f, 8 * h, lane);
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
          ff[f][k].h[h] = h0, ff[f][k].h[2 + h] = h1;
          ff[f][k].l[h] = l0, ff[f][k].l[2 + h] = l1;
        }
        if constexpr (FT) {
          uint32_t h0, l0;
          split2(y, both(cs), h0, l0);
          f8[f].h[h] = h0, f8[f].l[h] = l0;
        }
        __syncwarp();
      }
    }
    if (it + step < P.nit) codes(kn, code0, code1);

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
          float d[3][4] = {};
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            OpTile<uint4> b[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = oD[((c * KP + k) * NB + j) * 32];
            mma_tiles<PD>(d, fp[k], b, SET && k == 0);
          }
          if constexpr (KT) {
            OpTile<uint2> b[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = oDt[(c * NB + j) * 32];
            mma_tiles<PD>(d, fp8, b);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const bool lo = v < 2;
            const float *G = lo ? Ha : Hb;
            const float a = d[0][v], b = d[1][v], c = d[2][v];
#pragma unroll
            for (int x = 0; x < 3; ++x) rv[x][v] = G[x] * a + G[3 + x] * b + G[6 + x] * c;
          }
        }
        // a face's nodes are one step, k16 or k8 (N <= 4)
        static_assert(FP + FT == 1, "one step per face");
        float L[4][4];
        {
          OpTile<std::conditional_t<FT != 0, uint2, uint4>> b[4];
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            if constexpr (FT) b[f] = oLt[(f * NB + j) * 32];
            else b[f] = oL[(f * NB + j) * 32];
          }
#pragma unroll
          for (int p = 0; p < kProducts; ++p)
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              if constexpr (FT) mma_step<PR>(L[f], f8[f], b[f], p);
              else mma_step<PR>(L[f], ff[f][0], b[f], p);
            }
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
        // over the lane's own nodes in the p rows
        if (va) store4<Np, V>(Qa, n, make_float4(px[0], px[1], py[0], py[1]));
        if (vb) store4<Np, V>(Qb, n, make_float4(px[2], px[3], py[2], py[3]));
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
        if (va) store2<Np, V>(Qa, n, make_float2(px[0], px[1]));
        if (vb) store2<Np, V>(Qb, n, make_float2(px[2], px[3]));
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

    const float cma = __ldg(P.c2max + ka), cmb = __ldg(P.c2max + kb);
    // ---- 3. divergence of the contravariant velocities
    float r[NB][4];
    {
      // twice the bound: its own rounding cannot bring a value to 2^16
      const int sa = scale_field(2.f * Ma), sb = scale_field(2.f * Mb);
      const float ca = pow2_field(sa), cb = pow2_field(sb);
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          r[j][v] = 0.f;
        }
      // products of one operand step with the tiles b of all node blocks
      auto accumulate = [&](const auto &u, const auto B) {
        using T = decltype(B[0]);
#pragma unroll
        for (int j0 = 0; j0 < NB; j0 += 4) {
          constexpr int full = NB / 4 * 4, rem = NB % 4 ? NB % 4 : 4;
          if (j0 < full) {
            T b[4];
            float(&rr)[4][4] = *reinterpret_cast<float(*)[4][4]>(&r[j0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PD>(rr, u, b);
          } else {
            T b[rem];
            float(&rr)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(&r[j0]);
#pragma unroll
            for (int j = 0; j < rem; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PD>(rr, u, b);
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
      const float ia = -pow2_field(254 - sa) * P.iD, ib = -pow2_field(254 - sb) * P.iD;
      auto finish = [&](int j, const float (&l)[4]) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          r[j][v] = fmaf(r[j][v], v < 2 ? ia : ib, l[v]);
        }
      };
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const float4 a = load4<Np, V>(Qa, 16 * k + 4 * t), b = load4<Np, V>(Qb, 16 * k + 4 * t);
        const float l0[4] = {a.x, a.y, b.x, b.y}, l1[4] = {a.z, a.w, b.z, b.w};
        finish(2 * k, l0);
        finish(2 * k + 1, l1);
      }
      if constexpr (KT) {
        const float2 a = load2<Np, V>(Qa, 16 * KP + 2 * t), b = load2<Np, V>(Qb, 16 * KP + 2 * t);
        const float l[4] = {a.x, a.y, b.x, b.y};
        finish(2 * KP, l);
      }
    }
    __syncwarp();  // the tile is consumed: the next one on its way
    if (it + step < P.nit) fetch_tile(nshot, kn);

    // residual and old state of p, read while the projection runs
    const float *pa = Qs + ea, *pb = Qs + eb;
    float4 pra[KP > 0 ? KP : 1], prb[KP > 0 ? KP : 1], pqa[KP > 0 ? KP : 1], pqb[KP > 0 ? KP : 1];
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int n = 16 * k + 4 * t;
      pra[k] = load4<Np, V>(Ra, n), prb[k] = load4<Np, V>(Rb, n);
      pqa[k] = load4<Np, V>(pa, n), pqb[k] = load4<Np, V>(pb, n);
    }

    // ---- 4. WADG projection of rhs_p: 16 cubature points at a time through
    //         Vq, c2 and Pq
    float o[NB][4];
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
      const int wa = scale_field(P.vnorm * ma * cma),
                wb = scale_field(P.vnorm * mb * cmb);
      const float da = pow2_field(wa), db = pow2_field(wb);
      oia = pow2_field(254 - wa) * P.iP, oib = pow2_field(254 - wb) * P.iP;
      const float4 *Ca = reinterpret_cast<const float4 *>(P.c2p + (size_t)ka * P.Nq16) + t,
                   *Cb = reinterpret_cast<const float4 *>(P.c2p + (size_t)kb * P.Nq16) + t;
      const int nch = P.Nq16 / 16;
      float4 za = __ldg(Ca), zb = __ldg(Cb);  // c2 at this chunk's points
#pragma unroll 1
      for (int c = 0; c < nch; ++c) {
        float v[2][4] = {};
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          const OpTile<uint4> b[2] = {oV[((c * KP + k) * 2) * 32], oV[((c * KP + k) * 2 + 1) * 32]};
          mma_tiles<PR>(v, fr[k], b, SET && k == 0);
        }
        if constexpr (KT) {
          const OpTile<uint2> b[2] = {oVt[(c * 2) * 32], oVt[(c * 2 + 1) * 32]};
          mma_tiles<PR>(v, fr8, b);
        }
        // points 16 c + 4 t + 0 .. 3 of the two rows
        const float4 xa = make_float4(v[0][0] * via * za.x, v[0][1] * via * za.y,
                                      v[1][0] * via * za.z, v[1][1] * via * za.w);
        const float4 xb = make_float4(v[0][2] * vib * zb.x, v[0][3] * vib * zb.y,
                                      v[1][2] * vib * zb.z, v[1][3] * vib * zb.w);
        Frag w;
        split_frag(w, xa, xb, da, db);
        if (c + 1 < nch) za = __ldg(Ca + (c + 1) * 4), zb = __ldg(Cb + (c + 1) * 4);
        const O16 B = oP + c * NB * 32;
#pragma unroll
        for (int j0 = 0; j0 < NB; j0 += 4) {
          constexpr int full = NB / 4 * 4, rem = NB % 4 ? NB % 4 : 4;
          if (j0 < full) {
            OpTile<uint4> b[4];
            float(&oo)[4][4] = *reinterpret_cast<float(*)[4][4]>(&o[j0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(oo, w, b);
          } else {
            OpTile<uint4> b[rem];
            float(&oo)[rem][4] = *reinterpret_cast<float(*)[rem][4]>(&o[j0]);
#pragma unroll
            for (int j = 0; j < rem; ++j) b[j] = B[(j0 + j) * 32];
            mma_tiles<PR>(oo, w, b);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        o[j][v] *= v < 2 ? oia : oib;
      }

    // ---- 5. sources
    if (P.src_tile)
      tile_sources(P, Np, shot, k0, [&](int e, float amp, const float *vec) {
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const int n = j < 2 * KP ? 16 * (j / 2) + 4 * t + 2 * (j & 1) : 16 * KP + 2 * t;
          const float s0 = n < Np ? amp * __ldg(vec + n) : 0.f;
          const float s1 = n + 1 < Np ? amp * __ldg(vec + n + 1) : 0.f;
          if (e == g) o[j][0] += s0, o[j][1] += s1;
          if (e == g + 8) o[j][2] += s0, o[j][3] += s1;
        }
      });

    // ---- 6. LSRK update of p: res = fa res + fdt rhs, Q += fb res
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int n = 16 * k + 4 * t;
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
  WarpParams P = warp_params(pl, Qin, Qout, res, fa, fb, fdt, cstage);
  const int grid = warp_grid(pl, C::W, P);
  const size_t sm = warp_smem<N>(pl, pl.warp_ops);
  // split FP16 contexts (three products) exist from N = 2
  auto launch = [&](auto PR) {
    if (pl.warp_ops) k_warp_stage<N, decltype(PR)::value, true><<<grid, C::T, sm, st>>>(P);
    else k_warp_stage<N, decltype(PR)::value, false><<<grid, C::T, sm, st>>>(P);
  };
  if constexpr (N >= 2) {
    if (pl.products == 3) launch(std::integral_constant<int, 3>());
    else launch(std::integral_constant<int, 4>());
  } else {
    launch(std::integral_constant<int, 4>());
  }
  return check_launch("warp-matrix stage");
}

template <int N>
static bbw_status warp_prepare_n(WarpPlan &pl) {
  const int maxsm = device_smem_optin();
  pl.warp_ops = warp_smem<N>(pl, true) <= (size_t)maxsm;
  if (warp_smem<N>(pl, pl.warp_ops) > (size_t)maxsm)
    return set_error(BBW_ERR_UNSUPPORTED, "warp-matrix stage: does not fit in shared memory");
  if (N < 2 && pl.products == 3)
    return set_error(BBW_ERR_UNSUPPORTED, "warp-matrix stage: three products from N = 2");
  std::vector<const void *> fn = {(const void *)k_warp_stage<N, 4, false>,
                                  (const void *)k_warp_stage<N, 4, true>};
  if constexpr (N >= 2) {
    fn.push_back((const void *)k_warp_stage<N, 3, false>);
    fn.push_back((const void *)k_warp_stage<N, 3, true>);
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
