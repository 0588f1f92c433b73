// LSRK stage of the curved elements with every contraction on warp-level matrix
// instructions (warp_mma.cuh), a group of warps per 16-element tile.
//
// Replaces rk_volume_WADG_skew_combine + rk_surface_WADG_skew_combine +
// rk_update_WADG on curved elements (cpp/okl/WaveKernelsWADG.okl:514-682,
// 3024-3195, 1760-1887), as k_curved_stage (kernels_curved.cu) does with a thread
// per output: twenty Np x Nq contractions per element, and one operator load
// and one shared load per FMA there.  Here elements are matrix rows; operands
// are FP16 pairs scaled per element and field, operators pairs and a rest (the
// FP32 error, warp_mma.cuh),
// operator tiles come through L1 and the point values stay in registers.
#pragma once
#include "curved.h"
#include "warp_mma.cuh"

namespace bbw {

template <int N, int GWP>
struct CurvedCfg {
  static constexpr int Np = NP(N), Nfp = NFP(N), NF = 4 * NFP(N), EW = 4 * Np;
  static constexpr int NB = (Np + 7) / 8, KP = NB / 2, KT = NB % 2, U = KP + KT;
  static constexpr int FB = (Nfp + 7) / 8, FP = FB / 2, FT = FB % 2;
  // at most one unit of nodes per warp; 255 registers
  static constexpr int GW = GWP, NG = GW == 1 ? 6 : 8 / GW, T = 32 * GW * NG;
  static_assert(U <= GW, "a warp owns at most one unit");
  static constexpr int V = Np % 4 == 0 ? 4 : Np % 2 == 0 ? 2 : 1;
  static constexpr int AS = KP * 64 + KT * 32;              // uint4 of a split field
  // state rows, two of a pair 16 banks apart (as in group_stage.cuh), then four
  // split fields
  static constexpr int ODD = V == 4 ? (48 - EW % 32) % 32 : 0;
  __host__ __device__ static constexpr int row(int e) { return e * EW + ((e + 1) >> 1) * ODD; }
  static constexpr int ROWS = 16 * EW + 8 * ODD, TILE = ROWS > 16 * AS ? ROWS : 16 * AS;
  static constexpr int RC = N <= 3 ? 2 : 4;                 // cubature chunks per round
  static constexpr int WF = RC * 6 * 256;                   // split point values of a round
  static constexpr int MISC = GW * 64 + 2 * 4 * 16;         // maxima, two scales a face
  static int scratch(int FC) { return TILE + WF + MISC + 4 * FC * 4 * 256; }
};

template <int N, int GWP>
__global__ void __launch_bounds__(CurvedCfg<N, GWP>::T, 1)
    k_curved_mma(const CurvedMma A, const float *__restrict__ Qold, float *__restrict__ Qnew,
                 float *__restrict__ res) {
  using C = CurvedCfg<N, GWP>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NB = C::NB, KP = C::KP, KT = C::KT, EW = C::EW;
  constexpr int FP = C::FP, FT = C::FT, V = C::V, GW = C::GW, AS = C::AS, PR = 4, PD = 5;
  // a sum's first step sets it instead of adding to zero; by the registers (us per
  // stage added / set: N = 3, ball 24 107 / 105, N = 4, ball 12 50.7 / 46.1, N = 5, ball 10 54.7 / 56.0)
  constexpr bool SET = N == 3 || N == 4;
  extern __shared__ __align__(16) float smem_f[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = warp / GW, w = warp - grp * GW, g = lane >> 2, t = lane & 3;
  float *scr = smem_f + grp * A.scratch;
  float *sQ = scr;                                          // state rows, then
  uint4 *sA = reinterpret_cast<uint4 *>(scr);               // split p, u, v, w; then split rhs
  uint4 *sW = reinterpret_cast<uint4 *>(scr + C::TILE);     // split point values
  float4 *sMax = reinterpret_cast<float4 *>(scr + C::TILE + C::WF);  // [GW][16]
  float *sInv = scr + C::TILE + C::WF + GW * 64;            // [4][2][16] inverse flux scales
  uint4 *sFc = reinterpret_cast<uint4 *>(sInv + 128);       // [4][FC][4] split fluxes
  using O16 = Ops<uint4, PR, true>;
  using O8 = Ops<uint2, PR, true>;
  using T16 = OpTile<uint4>;
  auto op = [&](int off) { return O16(A.ops, A.ops + A.oM, off, lane); };
  auto tail = [&](int off) { return O8(A.ops, A.ops + A.oM, off, lane); };

  for (int it = blockIdx.x * C::NG + grp; it < A.nt; it += gridDim.x * C::NG) {
    const int r0 = it * 16, rl = A.KC - 1;
    const bool va = r0 + g < A.KC, vb = r0 + g + 8 < A.KC;
    const int ra_ = min(r0 + g, rl), rb_ = min(r0 + g + 8, rl);
    const size_t ea = (size_t)(A.k_off + ra_) * EW, eb = (size_t)(A.k_off + rb_) * EW;
    const float *Qa = sQ + C::row(ra_ - r0), *Qb = sQ + C::row(rb_ - r0);

    // ---- 0. state rows
    {
      const float4 *src = reinterpret_cast<const float4 *>(Qold + (size_t)(A.k_off + r0) * EW);
      const int ne = min(16, A.KC - r0);
      group_sync<GW>(grp);  // the previous tile's values are consumed
      for (int e = w; e < ne; e += GW)
#pragma unroll
        for (int c = lane; c < Np; c += 32)
          reinterpret_cast<float4 *>(sQ + C::row(e))[c] = __ldg(src + e * Np + c);
      group_sync<GW>(grp);
    }

    // ---- 1. faces: jumps and averages at the nodes, interpolated to the face
    //         cubature, upwind fluxes (rk_surface_WADG_skew_combine)
#pragma unroll 1
    for (int f = w; f < 4; f += GW) {
      constexpr int NV = FP * 4 + FT * 2;
      float x[7][2][NV];
      // pressure jumps, velocity jumps and averages may differ in size by any
      // factor (p ~ c u in the caller's units): a scale each
      float m[3] = {0.f, 0.f, 0.f}, mb[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = A.k_off + (h ? rb_ : ra_);
        const float *row = h ? Qb : Qa;
        const int *vm = A.vmapP + (size_t)k * C::NF + f * Nfp;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int i = j < FP * 4 ? 16 * (j / 4) + 4 * t + j % 4 : 16 * FP + 2 * t + j - FP * 4;
          const bool on = i < Nfp;
          const int nd = __ldg(A.Fmask + f * Nfp + (on ? i : 0)), idP = __ldg(vm + (on ? i : 0));
          const bool wall = idP == k * EW + nd;
          const float pM = row[nd], uM = row[Np + nd], vM = row[2 * Np + nd], wM = row[3 * Np + nd];
          const float pP = __ldg(Qold + idP), uP = __ldg(Qold + idP + Np),
                      vP = __ldg(Qold + idP + 2 * Np), wP = __ldg(Qold + idP + 3 * Np);
          x[0][h][j] = wall ? -2.f * pM : pP - pM;
          x[1][h][j] = uP - uM, x[2][h][j] = vP - vM, x[3][h][j] = wP - wM;
          x[4][h][j] = .5f * (uP + uM), x[5][h][j] = .5f * (vP + vM), x[6][h][j] = .5f * (wP + wM);
#pragma unroll
          for (int c = 0; c < 7; ++c) {
            if (!on) x[c][h][j] = 0.f;
            float &y = (h ? mb : m)[(c + 2) / 3];
            y = fmaxf(y, fabsf(x[c][h][j]));
          }
        }
      }
      float2 ca3[3], cb3[3];
      float ia[3], ib[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        m[q] = quad_max(m[q]), mb[q] = quad_max(mb[q]);
        const int sa = scale_field(m[q]), sb = scale_field(mb[q]);
        ca3[q] = both(pow2_field(sa)), cb3[q] = both(pow2_field(sb));
        ia[q] = pow2_field(254 - sa) * A.iF, ib[q] = pow2_field(254 - sb) * A.iF;
      }
      Frag fx[7][FP > 0 ? FP : 1];
      Frag8 f8[7];
#pragma unroll
      for (int c = 0; c < 7; ++c) {
        const float2 ca = ca3[(c + 2) / 3], cb = cb3[(c + 2) / 3];
#pragma unroll
        for (int s = 0; s < FP; ++s) {
          split2(make_float2(x[c][0][4 * s], x[c][0][4 * s + 1]), ca, fx[c][s].h[0], fx[c][s].l[0]);
          split2(make_float2(x[c][1][4 * s], x[c][1][4 * s + 1]), cb, fx[c][s].h[1], fx[c][s].l[1]);
          split2(make_float2(x[c][0][4 * s + 2], x[c][0][4 * s + 3]), ca, fx[c][s].h[2], fx[c][s].l[2]);
          split2(make_float2(x[c][1][4 * s + 2], x[c][1][4 * s + 3]), cb, fx[c][s].h[3], fx[c][s].l[3]);
        }
        if constexpr (FT) {
          split2(make_float2(x[c][0][4 * FP], x[c][0][4 * FP + 1]), ca, f8[c].h[0], f8[c].l[0]);
          split2(make_float2(x[c][1][4 * FP], x[c][1][4 * FP + 1]), cb, f8[c].h[1], f8[c].l[1]);
        }
      }
      // flux of p: |av - dp / 2| sJ <= fnorm (2 m[2] + m[0] / 2) sJ, of the velocities: |dp -
      // du| / 2 sJ <= fnorm (m[0] / 2 + m[1]) sJ (|n| = 1); twice that against rounding
      float da[2], db[2];
      {
        const float ka = 2.f * A.fnorm * __ldg(A.bound + (size_t)ra_ * 8 + 4 + f),
                    kb = 2.f * A.fnorm * __ldg(A.bound + (size_t)rb_ * 8 + 4 + f);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int ga = scale_field(ka * (q ? m[0] + m[1] : 2.f * m[2] + m[0])),
                    gb = scale_field(kb * (q ? mb[0] + mb[1] : 2.f * mb[2] + mb[0]));
          da[q] = pow2_field(ga), db[q] = pow2_field(gb);
          if (t == 0) {
            sInv[(f * 2 + q) * 16 + g] = pow2_field(254 - ga) * A.iP;
            sInv[(f * 2 + q) * 16 + g + 8] = pow2_field(254 - gb) * A.iP;
          }
        }
      }
#pragma unroll 1
      for (int ch = 0; ch < A.FC; ++ch) {
        float v[7][2][4];
        auto each = [&](float (&o)[7][4], const auto &x, const auto b) {
#pragma unroll
          for (int p = 0; p < kProducts; ++p)
#pragma unroll
            for (int c = 0; c < 7; ++c) mma_step<PR>(o[c], x(c), b, p);
        };
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float s7[7][4];
#pragma unroll
          for (int s = 0; s < FP; ++s) {
            each(s7, [&](int c) { return fx[c][s]; }, op(A.oF)[((ch * FP + s) * 2 + i) * 32]);
#pragma unroll
            for (int c = 0; c < 7; ++c) add4(v[c][i], s7[c], s == 0);
          }
          if constexpr (FT) {
            each(s7, [&](int c) { return f8[c]; }, tail(A.oFt)[(ch * 2 + i) * 32]);
#pragma unroll
            for (int c = 0; c < 7; ++c) add4(v[c][i], s7[c], FP == 0);
          }
        }
        // points 16 ch + 4 t + 0 .. 3: row h, point 2 i + j of the four
        float fl[4][2][4];
        const float *G = A.fq + ((size_t)(it * 4 + f) * A.FC + ch) * 4 * 256;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 *gp = reinterpret_cast<const float4 *>(G + (g + 8 * h) * 16) + t;
          const float4 n0 = __ldg(gp), n1 = __ldg(gp + 64), n2 = __ldg(gp + 128), n3 = __ldg(gp + 192);
          const float nx[4] = {n0.x, n0.y, n0.z, n0.w}, ny[4] = {n1.x, n1.y, n1.z, n1.w};
          const float nz[4] = {n2.x, n2.y, n2.z, n2.w}, sJ[4] = {n3.x, n3.y, n3.z, n3.w};
          const float *inv = h ? ib : ia;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = q / 2, j = 2 * h + q % 2;
            const float dp = v[0][i][j] * inv[0];
            const float uj = (v[1][i][j] * nx[q] + v[2][i][j] * ny[q] + v[3][i][j] * nz[q]) * inv[1];
            const float ua = (v[4][i][j] * nx[q] + v[5][i][j] * ny[q] + v[6][i][j] * nz[q]) * inv[2];
            const float U = -.5f * (dp - uj) * sJ[q];
            fl[0][h][q] = -(ua - .5f * dp) * sJ[q];
            fl[1][h][q] = U * nx[q], fl[2][h][q] = U * ny[q], fl[3][h][q] = U * nz[q];
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          Frag o;
          split_frag(o, make_float4(fl[c][0][0], fl[c][0][1], fl[c][0][2], fl[c][0][3]),
                     make_float4(fl[c][1][0], fl[c][1][1], fl[c][1][2], fl[c][1][3]), da[c > 0], db[c > 0]);
          put_frag(sFc + ((f * A.FC + ch) * 4 + c) * 64, 0, lane, o);
        }
      }
    }

    // ---- 2. split p, u, v, w (over the rows)
    float4 qa[4], qb[4];  // the warp's unit of the old state
    const bool mine = w < C::U, pair = w < KP;  // a unit of this warp; of two blocks
    float sc[4][2];       // scales, later inverse scales
    auto maxima = [&](const float4 (&xa)[4], const float4 (&xb)[4]) {
      float m[8];
#pragma unroll
      for (int c = 0; c < 4; ++c) m[c] = quad_max(max4(0.f, xa[c])), m[4 + c] = quad_max(max4(0.f, xb[c]));
      if (t < 2) sMax[w * 16 + g + 8 * t] = t == 0 ? make_float4(m[0], m[1], m[2], m[3])
                                                 : make_float4(m[4], m[5], m[6], m[7]);
    };
    float4 ma, mb;
    auto read_maxima = [&]() {
      ma = sMax[g], mb = sMax[g + 8];
#pragma unroll
      for (int i = 1; i < GW; ++i) {
        const float4 a = sMax[i * 16 + g], b = sMax[i * 16 + g + 8];
        ma = make_float4(fmaxf(ma.x, a.x), fmaxf(ma.y, a.y), fmaxf(ma.z, a.z), fmaxf(ma.w, a.w));
        mb = make_float4(fmaxf(mb.x, b.x), fmaxf(mb.y, b.y), fmaxf(mb.z, b.z), fmaxf(mb.w, b.w));
      }
    };
    // fields xa, xb of the warp's unit to sA, scaled by sc
    auto split_unit = [&](const float4 (&xa)[4], const float4 (&xb)[4]) {
      if (!mine) return;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (pair) {
          Frag f;
          split_frag(f, xa[c], xb[c], sc[c][0], sc[c][1]);
          put_frag(sA + c * AS, w, lane, f);
        } else {
          Frag8 f;
          split_frag(f, lo2(xa[c]), lo2(xb[c]), sc[c][0], sc[c][1]);
          put_frag8(sA + c * AS, KP, lane, f);
        }
      }
    };
    auto set_scales = [&]() {  // sc from the maxima; returns nothing, inverse by invert()
      const float a[4] = {ma.x, ma.y, ma.z, ma.w}, b[4] = {mb.x, mb.y, mb.z, mb.w};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        sc[c][0] = pow2_field(scale_field(a[c])), sc[c][1] = pow2_field(scale_field(b[c]));
    };
    auto load_unit = [&](const float *p, int c) {
      if (!mine) return make_float4(0.f, 0.f, 0.f, 0.f);
      if (pair) return load4<Np, V>(p + c * Np, 16 * w + 4 * t);
      const float2 y = load2<Np, V>(p + c * Np, 16 * KP + 2 * t);
      return make_float4(y.x, y.y, 0.f, 0.f);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) qa[c] = load_unit(Qa, c), qb[c] = load_unit(Qb, c);
    maxima(qa, qb);
    group_sync<GW>(grp);  // maxima and fluxes ready, the rows are read
    read_maxima();
    set_scales();
    split_unit(qa, qb);
    group_sync<GW>(grp);

    // ---- 3. volume terms (rk_volume_WADG_skew_combine): J grad p and -J times
    //         the contravariant velocities at the cubature, projected
    float r[4][2][4];  // rhs of the warp's unit
    {
      const float um = fmaxf(fmaxf(ma.y, ma.z), ma.w), un = fmaxf(fmaxf(mb.y, mb.z), mb.w);
      const float *Ba = A.bound + (size_t)ra_ * 8, *Bb = A.bound + (size_t)rb_ * 8;
      // gradient of p (for u, v, w) and contravariant velocities (for p): a scale each
      const int ta[2] = {scale_field(2.f * __ldg(Ba) * A.dnorm * ma.x),
                         scale_field(2.f * __ldg(Ba + 1) * A.vnorm * um)};
      const int tb[2] = {scale_field(2.f * __ldg(Bb) * A.dnorm * mb.x),
                         scale_field(2.f * __ldg(Bb + 1) * A.vnorm * un)};
      float isc[4][2];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) isc[c][h] = (1.f / sc[c][h]) * (c == 0 ? A.iD : A.iV);
      float o[4][2][4] = {};
#pragma unroll 1
      for (int c0 = 0; c0 < A.nch; c0 += C::RC) {
        const int cend = min(A.nch, c0 + C::RC);
        if (c0 > 0) group_sync<GW>(grp);
#pragma unroll 1
        for (int c = c0 + w; c < cend; c += GW) {
          // u, v, w with Vq; p with Vrq, Vsq, Vtq
          float v[6][2][4] = {};
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            const Frag p = get_frag(sA, k, lane);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const O16 D = op(A.oV[1 + d]) + ((c * KP + k) * 2) * 32;
              const O16 Q = op(A.oV[0]) + ((c * KP + k) * 2) * 32;
              const T16 bd[2] = {D[0], D[32]}, bq[2] = {Q[0], Q[32]};
              const Frag u = get_frag(sA + (1 + d) * AS, k, lane);
              mma_pair2<PD, PR>(v[3 + d], p, bd, v[d], u, bq, SET && k == 0, SET && k == 0);
            }
          }
          if constexpr (KT) {
            const Frag8 p = get_frag8(sA, KP, lane);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const O8 D = tail(A.oVt[1 + d]) + (c * 2) * 32, Q = tail(A.oVt[0]) + (c * 2) * 32;
              const OpTile<uint2> bd[2] = {D[0], D[32]}, bq[2] = {Q[0], Q[32]};
              const Frag8 u = get_frag8(sA + (1 + d) * AS, KP, lane);
              mma_pair2<PD, PR>(v[3 + d], p, bd, v[d], u, bq);
            }
          }
          const float *G = A.gq + ((size_t)it * A.nch + c) * 10 * 256;
          float4 tv[6][2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 *gp = reinterpret_cast<const float4 *>(G + (g + 8 * h) * 16) + t;
            float G9[10][4];
#pragma unroll
            for (int i = 0; i < 10; ++i) {
              const float4 y = __ldg(gp + 64 * i);
              G9[i][0] = y.x, G9[i][1] = y.y, G9[i][2] = y.z, G9[i][3] = y.w;
            }
            float o6[6][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = q / 2, j = 2 * h + q % 2;
              const float uq = v[0][i][j] * isc[1][h], vq = v[1][i][j] * isc[2][h],
                          wq = v[2][i][j] * isc[3][h];
              const float dr = v[3][i][j] * isc[0][h], ds = v[4][i][j] * isc[0][h],
                          dt = v[5][i][j] * isc[0][h];
              const float J = G9[9][q];
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                // vgeoq order rx sx tx ry sy ty rz sz tz
                o6[x][q] = (G9[3 * x][q] * dr + G9[3 * x + 1][q] * ds + G9[3 * x + 2][q] * dt) * J;
                o6[3 + x][q] = -((uq * G9[x][q] + vq * G9[3 + x][q] + wq * G9[6 + x][q]) * J);
              }
            }
#pragma unroll
            for (int x = 0; x < 6; ++x) tv[x][h] = make_float4(o6[x][0], o6[x][1], o6[x][2], o6[x][3]);
          }
#pragma unroll
          for (int x = 0; x < 6; ++x) {
            Frag f;
            split_frag(f, tv[x][0], tv[x][1], pow2_field(ta[x / 3]), pow2_field(tb[x / 3]));
            put_frag(sW + ((c - c0) * 6 + x) * 64, 0, lane, f);
          }
        }
        group_sync<GW>(grp);
#pragma unroll 1
        for (int c = c0; c < cend && mine; ++c) {
          const uint4 *W = sW + (c - c0) * 6 * 64;
          const int at = (c * NB + 2 * w) * 32;
          // field p (o[0]) collects Prq, Psq, Ptq; u, v, w take Pq
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const Frag x = get_frag(W + d * 64, 0, lane), y = get_frag(W + (3 + d) * 64, 0, lane);
            const O16 Q = op(A.oP[0]) + at, D = op(A.oP[1 + d]) + at;
            if (pair) {
              const T16 bq[2] = {Q[0], Q[32]}, bd[2] = {D[0], D[32]};
              mma_pair2<PR, PD>(o[1 + d], x, bq, o[0], y, bd);
            } else {
              const T16 bq[1] = {Q[0]}, bd[1] = {D[0]};
              mma_pair2<PR, PD>(one(o[1 + d]), x, bq, one(o[0]), y, bd);
            }
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float ia = -pow2_field(254 - ta[c == 0]) * A.iP, ib = -pow2_field(254 - tb[c == 0]) * A.iP;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) r[c][i][j] = o[c][i][j] * (j < 2 ? ia : ib);
      }
    }

    // ---- 4. lifted fluxes
#pragma unroll 1
    for (int f = 0; f < 4 && mine; ++f) {
      float o[4][2][4] = {};
#pragma unroll 1
      for (int ch = 0; ch < A.FC; ++ch) {
        const uint4 *W = sFc + (f * A.FC + ch) * 4 * 64;
        const O16 B = op(A.oL) + ((f * A.FC + ch) * NB + 2 * w) * 32;
        const T16 b[2] = {B[0], B[pair ? 32 : 0]};
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          const Frag x = get_frag(W + c * 64, 0, lane), y = get_frag(W + (c + 1) * 64, 0, lane);
          if (pair) {
            mma_pair2<PR, PR>(o[c], x, b, o[c + 1], y, b);
          } else {
            const T16 b1[1] = {b[0]};
            mma_pair2<PR, PR>(one(o[c]), x, b1, one(o[c + 1]), y, b1);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            r[c][i][j] = fmaf(o[c][i][j], sInv[(f * 2 + (c > 0)) * 16 + g + (j < 2 ? 0 : 8)], r[c][i][j]);
    }

    // ---- 5. rk_update_WADG: interpolate, weight with 1/J (c2/J on p), project
    {
      float4 xa[4], xb[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (pair) {
          xa[c] = make_float4(r[c][0][0], r[c][0][1], r[c][1][0], r[c][1][1]);
          xb[c] = make_float4(r[c][0][2], r[c][0][3], r[c][1][2], r[c][1][3]);
        } else {
          xa[c] = make_float4(r[c][0][0], r[c][0][1], 0.f, 0.f);
          xb[c] = make_float4(r[c][0][2], r[c][0][3], 0.f, 0.f);
        }
      }
      maxima(xa, xb);
      group_sync<GW>(grp);  // maxima ready; the split state is consumed
      read_maxima();
      set_scales();
      split_unit(xa, xb);
      group_sync<GW>(grp);
    }
    float o[4][2][4] = {};
    float oinv[4][2];
    {
      float isc[4][2], d[4][2];
      const float *Ba = A.bound + (size_t)ra_ * 8, *Bb = A.bound + (size_t)rb_ * 8;
      const float a[4] = {ma.x, ma.y, ma.z, ma.w}, b[4] = {mb.x, mb.y, mb.z, mb.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // |Vq r| / J <= vnorm max|r| max 1/J (times c2 on p)
        const int fa = scale_field(2.f * A.rnorm * a[c] * __ldg(Ba + (c == 0 ? 2 : 3))),
                  fb = scale_field(2.f * A.rnorm * b[c] * __ldg(Bb + (c == 0 ? 2 : 3)));
        d[c][0] = pow2_field(fa), d[c][1] = pow2_field(fb);
        oinv[c][0] = pow2_field(254 - fa) * A.iPr, oinv[c][1] = pow2_field(254 - fb) * A.iPr;
        isc[c][0] = (1.f / sc[c][0]) * A.iVr, isc[c][1] = (1.f / sc[c][1]) * A.iVr;
      }
#pragma unroll 1
      for (int c0 = 0; c0 < A.nchr; c0 += C::RC) {
        const int cend = min(A.nchr, c0 + C::RC);
        if (c0 > 0) group_sync<GW>(grp);
#pragma unroll 1
        for (int c = c0 + w; c < cend; c += GW) {
          float v[4][2][4] = {};
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            const O16 B = op(A.oVr) + ((c * KP + k) * 2) * 32;
            const T16 b2[2] = {B[0], B[32]};
#pragma unroll
            for (int x = 0; x < 4; x += 2)
              mma_pair2<PR, PR>(v[x], get_frag(sA + x * AS, k, lane), b2, v[x + 1],
                            get_frag(sA + (x + 1) * AS, k, lane), b2, SET && k == 0, SET && k == 0);
          }
          if constexpr (KT) {
            const O8 B = tail(A.oVrt) + (c * 2) * 32;
            const OpTile<uint2> b2[2] = {B[0], B[32]};
#pragma unroll
            for (int x = 0; x < 4; x += 2)
              mma_pair2<PR, PR>(v[x], get_frag8(sA + x * AS, KP, lane), b2, v[x + 1],
                            get_frag8(sA + (x + 1) * AS, KP, lane), b2);
          }
          const float *G = A.jq + ((size_t)it * A.nchr + c) * 2 * 256;
          const float4 *pa = reinterpret_cast<const float4 *>(G + g * 16) + t, *pb = pa + 32;
          const float4 ja = __ldg(pa), jb = __ldg(pb), za = __ldg(pa + 64), zb = __ldg(pb + 64);
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            float4 ya = make_float4(v[x][0][0] * isc[x][0] * ja.x,
                                    v[x][0][1] * isc[x][0] * ja.y,
                                    v[x][1][0] * isc[x][0] * ja.z,
                                    v[x][1][1] * isc[x][0] * ja.w);
            float4 yb = make_float4(v[x][0][2] * isc[x][1] * jb.x,
                                    v[x][0][3] * isc[x][1] * jb.y,
                                    v[x][1][2] * isc[x][1] * jb.z,
                                    v[x][1][3] * isc[x][1] * jb.w);
            if (x == 0) {
              ya = make_float4(ya.x * za.x, ya.y * za.y, ya.z * za.z, ya.w * za.w);
              yb = make_float4(yb.x * zb.x, yb.y * zb.y, yb.z * zb.z, yb.w * zb.w);
            }
            Frag f;
            split_frag(f, ya, yb, d[x][0], d[x][1]);
            put_frag(sW + ((c - c0) * 4 + x) * 64, 0, lane, f);
          }
        }
        group_sync<GW>(grp);
#pragma unroll 1
        for (int c = c0; c < cend && mine; ++c) {
          const uint4 *W = sW + (c - c0) * 4 * 64;
          const O16 B = op(A.oPr) + (c * NB + 2 * w) * 32;
          const T16 b2[2] = {B[0], B[pair ? 32 : 0]};
#pragma unroll
          for (int x = 0; x < 4; x += 2) {
            const Frag f0 = get_frag(W + x * 64, 0, lane), f1 = get_frag(W + (x + 1) * 64, 0, lane);
            if (pair) {
              mma_pair2<PR, PR>(o[x], f0, b2, o[x + 1], f1, b2);
            } else {
              const T16 b1[1] = {b2[0]};
              mma_pair2<PR, PR>(one(o[x]), f0, b1, one(o[x + 1]), f1, b1);
            }
          }
        }
      }
    }

    // ---- 6. res = fa res + dt r, Q = Q + fb res
    const float2 fa2 = both(A.fa), fd2 = both(A.fdt), fb2 = both(A.fb);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const size_t at = (h ? eb : ea) + c * Np;
        const float s = oinv[c][h];
        const float4 q = h ? qb[c] : qa[c];
        if (!mine || !(h ? vb : va)) continue;
        const float2 x0 = make_float2(o[c][0][2 * h] * s,
                                      o[c][0][2 * h + 1] * s);
        if (pair) {
          const float2 x1 = make_float2(o[c][1][2 * h] * s,
                                        o[c][1][2 * h + 1] * s);
          const int n = 16 * w + 4 * t;
          const float4 old = load4<Np, V>(res + at, n);
          const float2 y0 = lsrk2(lo2(old), x0, fa2, fd2), y1 = lsrk2(hi2(old), x1, fa2, fd2);
          const float2 z0 = __ffma2_rn(fb2, y0, lo2(q)), z1 = __ffma2_rn(fb2, y1, hi2(q));
          store4<Np, V>(res + at, n, make_float4(y0.x, y0.y, y1.x, y1.y));
          store4<Np, V>(Qnew + at, n, make_float4(z0.x, z0.y, z1.x, z1.y));
        } else {
          const int n = 16 * KP + 2 * t;
          const float2 y = lsrk2(load2<Np, V>(res + at, n), x0, fa2, fd2);
          store2<Np, V>(res + at, n, y);
          store2<Np, V>(Qnew + at, n, __ffma2_rn(fb2, y, lo2(q)));
        }
      }
  }
}

template <int N, int GW>
static bbw_status curved_mma_launch_g(const CurvedMma &A, const float *Qold, float *Qnew, float *res,
                                      cudaStream_t st) {
  using C = CurvedCfg<N, GW>;
  CurvedMma P = A;
  P.scratch = C::scratch(A.FC);
  const size_t sm = sizeof(float) * (size_t)C::NG * P.scratch;
  const int need = (A.nt + C::NG - 1) / C::NG, grid = need < A.nsm ? need : A.nsm;
  k_curved_mma<N, GW><<<grid, C::T, sm, st>>>(P, Qold, Qnew, res);
  return check_launch("curved matrix stage");
}

template <int N, int GW>
static bbw_status curved_mma_prepare_g(const CurvedMma &A) {
  using C = CurvedCfg<N, GW>;
  const int maxsm = device_smem_optin();
  if (sizeof(float) * (size_t)C::NG * C::scratch(A.FC) > (size_t)maxsm)
    return set_error(BBW_ERR_UNSUPPORTED, "curved matrix stage: does not fit in shared memory");
  return ensure_smem_limit((const void *)k_curved_mma<N, GW>, maxsm, "curved matrix stage attribute");
}

// Warps per tile: four (a face each) while the tiles fit one wave of two
// groups per SM, else as many as there are units of nodes (the results are the
// same).  us per stage with the planar elements, N = 3, before the rests: K = 3072
// (84 tiles) 21.2 with four, 24.9 with two; K = 82944 (828 tiles) 114 and 99.
template <int N>
static bool curved_wide(const CurvedMma &A) { return A.nt <= 2 * A.nsm; }

template <int N>
static bbw_status curved_mma_launch_n(const CurvedMma &A, const float *Qold, float *Qnew, float *res,
                                      cudaStream_t st) {
  constexpr int GW = N <= 2 ? 1 : N == 3 ? 2 : 4;
  if (GW == 4 || curved_wide<N>(A)) return curved_mma_launch_g<N, 4>(A, Qold, Qnew, res, st);
  return curved_mma_launch_g<N, GW>(A, Qold, Qnew, res, st);
}

template <int N>
static bbw_status curved_mma_prepare_n(const CurvedMma &A) {
  constexpr int GW = N <= 2 ? 1 : N == 3 ? 2 : 4;
  const bbw_status s = curved_mma_prepare_g<N, 4>(A);
  return s != BBW_OK || GW == 4 ? s : curved_mma_prepare_g<N, GW>(A);
}

#define BBW_CURVED_MMA_INSTANCE(n)                                                                \
  bbw_status curved_mma_launch_##n(const CurvedMma &A, const float *Qold, float *Qnew, float *res, \
                                   cudaStream_t st) {                                             \
    return curved_mma_launch_n<n>(A, Qold, Qnew, res, st);                                        \
  }                                                                                               \
  bbw_status curved_mma_prepare_##n(const CurvedMma &A) { return curved_mma_prepare_n<n>(A); }

}  // namespace bbw
