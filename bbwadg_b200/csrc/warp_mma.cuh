// Shared pieces of the stages on warp-level matrix instructions (warp_stage.cuh,
// group_stage.cuh): mma.sync m16n8k16 on FP16 pairs with FP32 accumulation.
//
// Elements are the rows (M = 16) of every product and operator rows the
// columns, so the accumulators of one contraction have the register layout of
// the next one's A operand.  mma.sync gives 1024 FMA per cycle and SM here (8
// cycles per m16n8k16 and SM quarter, measured; k8 costs the same), a quarter of
// what tcgen05 does on full tiles, with a latency of 21 cycles and no TMEM
// round trip: the contractions are skinny (K = Np, Nfp or Nq per element), and
// the chain of dependent phases bounds them, not the tensor rate.
//
// FP32 values x are split into FP16 pairs x s = hi + lo with a power of two s
// per element and operand, so each element keeps its own dynamic range.  A pair
// holds 23 bits: one short of FP32.  For the operand that is a rounding that
// changes from stage to stage; for an operator it would be the same error in
// every stage, which a time loop adds up, so operators keep a third part (the
// rest, a byte of three significant bits: 26 bits in all).  Likewise the matrix
// unit's rounding toward zero, see mma_step.  Error after 100 stages over the
// CUDA-core stage's, pairs alone and summed in one accumulator / this form
// (relative L2 against 64 bits, mean of 14 smooth states): N = 2 1.13 / 0.97, N = 4
// 1.12 / 1.02, N = 5 1.28 / 1.01, BB 1.32 / 0.97, N = 6 1.32 / 1.01, each to 2 %; of one
// right-hand side 0.8 .. 1.1.  The split-FP16 form has no rest and takes three products.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "device_common.cuh"
#include "warp_stage.h"

namespace bbw {

struct WarpParams {
  int K, K0, Kc, Nq, Nq16, bc, pat_off, table_ints, bs, ws, nt32;
  int nit, ntile, step_shot, step_tile;  // items; tiles per shot; a group's stride in both
  int oDt, oL, oLt, oV, oVt, oP, oM, ops_n;  // operator offsets and size in uint4
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
  const double *time;
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

// the same with nothing to add to
__device__ __forceinline__ void mma16_set(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ void mma8_set(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%7,%7,%7,%7};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(0.f));
}

// c = s (the first step), or c += s, rounded to nearest
__device__ __forceinline__ void add4(float (&c)[4], const float (&s)[4], bool first = false) {
  if (first) {
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = s[i];
    return;
  }
  const float2 a = __fadd2_rn(make_float2(c[0], c[1]), make_float2(s[0], s[1]));
  const float2 b = __fadd2_rn(make_float2(c[2], c[3]), make_float2(s[2], s[3]));
  c[0] = a.x, c[1] = a.y, c[2] = b.x, c[3] = b.y;
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

// Operator tile of a k16 (W = uint4) or k8 step (uint2): the lane's hi and lo
// words, and the bytes of the rest (four-product forms)
template <class W>
struct OpTile {
  W w;
  uint32_t m;
};
// Tiles in memory; the rests are a plane of their own, a byte per four of the
// words.  GW, GM: words, rests in global memory (read-only path), else in shared.
template <class W, int PR, bool GW, bool GM = GW>
struct Ops {
  using M = std::conditional_t<sizeof(W) == 16, uint32_t, uint16_t>;
  const W *w;
  const M *m;
  // at: uint4 offset of the lane's first tile in the words at ops
  __device__ __forceinline__ Ops(const uint4 *ops, const void *rests, int at, int lane)
      : w(reinterpret_cast<const W *>(ops + at) + lane),
        m(reinterpret_cast<const M *>(rests) + at * (int)(16 / sizeof(W)) + lane) {}
  __device__ __forceinline__ Ops(const W *a, const M *b) : w(a), m(b) {}
  __device__ __forceinline__ Ops operator+(int i) const { return Ops(w + i, m + i); }
  __device__ __forceinline__ OpTile<W> operator[](int i) const {
    OpTile<W> t;
    if constexpr (GW) t.w = __ldg(w + i);
    else t.w = w[i];
    if constexpr (PR < 4) t.m = 0;
    else if constexpr (GM) t.m = __ldg(m + i);
    else t.m = m[i];
    return t;
  }
};
// two bytes of the rest as FP16 pairs
__device__ __forceinline__ uint32_t rest_lo(uint32_t m) { return __byte_perm(m, 0, 0x1404); }
__device__ __forceinline__ uint32_t rest_hi(uint32_t m) { return __byte_perm(m, 0, 0x3424); }

// One k step of a contraction is summed from zero and added to the result on
// the CUDA cores (add4).  The matrix unit rounds its sums toward zero: a chain of
// steps in one accumulator loses half an ulp of the running sum at every step,
// always the same way.  One such rounding per step is left, and the operators
// are packed larger by its mean (kRoundingBias).  us per stage against one
// accumulator, N = 5, K = 196608: 411 -> 432; N = 7, K = 24576: 177 -> 212.
//
// Product p of one step, from zero or onto s, smallest first: the operand's hi
// with the operator's rest, lo with lo, hi with lo, lo with hi, hi with hi.  PR = 5:
// all; 4: without lo with lo; 3: the last three.  A k8 step takes two of them in
// one k16 product, which costs no more, so there 4 is 5.
constexpr int kProducts = 5;
template <int PR>
__device__ __forceinline__ void mma_step(float (&s)[4], const Frag &x, const OpTile<uint4> &b, int p) {
  if constexpr (PR >= 4) {
    if (p == 0) mma16_set(s, x.h, rest_lo(b.m), rest_hi(b.m));
    if (p == 1 && PR == 5) mma16(s, x.l, b.w.z, b.w.w);
    if (p == 2) mma16(s, x.h, b.w.z, b.w.w);
  } else if (p == 2) {
    mma16_set(s, x.h, b.w.z, b.w.w);
  }
  if (p == 3) mma16(s, x.l, b.w.x, b.w.y);
  if (p == 4) mma16(s, x.h, b.w.x, b.w.y);
}
template <int PR>
__device__ __forceinline__ void mma_step(float (&s)[4], const Frag8 &x, const OpTile<uint2> &b, int p) {
  const uint32_t hl[4] = {x.h[0], x.h[1], x.l[0], x.l[1]};
  if constexpr (PR >= 4) {
    if (p == 0) mma16_set(s, hl, rest_lo(b.m), b.w.y);
    if (p == 2) mma16(s, hl, b.w.y, b.w.x);
  } else if (p == 2) {
    mma16_set(s, hl, b.w.y, b.w.x);
  }
  if (p == 4) mma8(s, x.h[0], x.h[1], b.w.x);
}

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

// c += x b (first: c = x b) for M operator tiles; an accumulator is used again only after the
// other tiles' product (a product takes 21 cycles, 8 of them issuing)
template <int PR, int M, class F, class T>
__device__ __forceinline__ void mma_tiles(float (&c)[M][4], const F &x, const T (&b)[M], bool first = false) {
  float s[M][4];
#pragma unroll
  for (int p = 0; p < kProducts; ++p)
#pragma unroll
    for (int i = 0; i < M; ++i) mma_step<PR>(s[i], x, b[i], p);
#pragma unroll
  for (int i = 0; i < M; ++i) add4(c[i], s[i], first);
}
// the first of two accumulators as an array of one
__device__ __forceinline__ float (&one(float (&c)[2][4]))[1][4] {
  return *reinterpret_cast<float(*)[1][4]>(&c[0]);
}
template <int PR, class F, class T>
__device__ __forceinline__ void mma_tile(float (&c)[4], const F &x, const T b) {
  const T b1[1] = {b};
  mma_tiles<PR>(*reinterpret_cast<float(*)[1][4]>(&c), x, b1);
}
// two operands' products x b and y bb, interleaved
template <int PX, int PY, int M, class F, class T>
__device__ __forceinline__ void mma_pair2(float (&c)[M][4], const F &x, const T (&b)[M],
                                          float (&cc)[M][4], const F &y, const T (&bb)[M],
                                          bool first = false, bool first2 = false) {
  float s[M][4], ss[M][4];
#pragma unroll
  for (int p = 0; p < kProducts; ++p) {
#pragma unroll
    for (int i = 0; i < M; ++i) mma_step<PX>(s[i], x, b[i], p);
#pragma unroll
    for (int i = 0; i < M; ++i) mma_step<PY>(ss[i], y, bb[i], p);
  }
#pragma unroll
  for (int i = 0; i < M; ++i) add4(c[i], s[i], first);
#pragma unroll
  for (int i = 0; i < M; ++i) add4(cc[i], ss[i], first2);
}

// index of slot c of block b when n indices are stored in blocks of eight
// (warp_stage.h)
__device__ __forceinline__ int slot_index(int n, int b, int c) {
  const int nb = (n + 7) / 8;
  if (b == nb - 1 && nb % 2) return 8 * b + c;
  return 16 * (b / 2) + 4 * (c / 2) + 2 * (b % 2) + c % 2;
}

// two operator values as hi, lo and the bytes of the rest, larger by
// kRoundingBias
__device__ __forceinline__ void split_operator(float2 x, float s, uint32_t &h, uint32_t &l, uint32_t &m) {
  const float2 y = __fmul2_rn(x, both(s));
  const __half2 hh = __float22half2_rn(y);
  const float2 f = __half22float2(hh);
  const float2 r = __ffma2_rn(y, both((float)kRoundingBias), __fadd2_rn(y, make_float2(-f.x, -f.y)));
  const __half2 ll = __float22half2_rn(r);
  const float2 g = __half22float2(ll);
  const __half2 mm = __float22half2_rn(__fadd2_rn(r, make_float2(-g.x, -g.y)));
  h = *reinterpret_cast<const uint32_t *>(&hh);
  l = *reinterpret_cast<const uint32_t *>(&ll);
  m = rest_byte(__half_as_ushort(__low2half(mm))) | rest_byte(__half_as_ushort(__high2half(mm))) << 8;
}
// lane's words of a k16 (uint4) or k8 (uint2) tile and its rest (null: none): at(block,
// slot) gives the entries
template <bool K16, class At>
__device__ __forceinline__ void split_tile(uint32_t *out, uint32_t *rest, int i, int k, int c, float s,
                                           At &&at) {
  uint32_t h0, l0, m0;
  if constexpr (K16) {
    uint32_t h1, l1, m1;
    split_operator(make_float2(at(2 * k, c), at(2 * k, c + 1)), s, h0, l0, m0);
    split_operator(make_float2(at(2 * k + 1, c), at(2 * k + 1, c + 1)), s, h1, l1, m1);
    reinterpret_cast<uint4 *>(out)[i] = make_uint4(h0, h1, l0, l1);
    if (rest) rest[i] = m0 | m1 << 16;
  } else {
    split_operator(make_float2(at(k, c), at(k, c + 1)), s, h0, l0, m0);
    reinterpret_cast<uint2 *>(out)[i] = make_uint2(h0, l0);
    if (rest) reinterpret_cast<uint16_t *>(rest)[i] = (uint16_t)m0;
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

// A value of a neighbour's state.  CHAINED: by the coherent path, as the stage
// before may still run when this kernel starts; not volatile, so that loads
// schedule freely: the address comes from a table that is read after stage_wait.
template <bool CHAINED>
__device__ __forceinline__ float load_trace(const float *x) {
  if constexpr (!CHAINED) return __ldg(x);
  float v;
  asm("ld.global.f32 %0, [%1];\n" : "=f"(v) : "l"(x));
  return v;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
// n uint4 to shared memory by T threads
template <int T>
__device__ __forceinline__ void stage_async(uint4 *dst, const uint4 *src, int n) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += T) cp_async16(d + 16 * i, reinterpret_cast<const float *>(src + i));
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

// res = fa res + fdt rhs, Q += fb res for four values
__device__ __forceinline__ void lsrk4(const float4 r0, const float4 x, const float4 q0,
                                      const WarpParams &P, float4 &r, float4 &q) {
  const float2 a = lsrk2(lo2(r0), lo2(x), both(P.fa), both(P.fdt));
  const float2 b = lsrk2(hi2(r0), hi2(x), both(P.fa), both(P.fdt));
  const float2 c = __ffma2_rn(both(P.fb), a, lo2(q0)), d = __ffma2_rn(both(P.fb), b, hi2(q0));
  r = make_float4(a.x, a.y, b.x, b.y), q = make_float4(c.x, c.y, d.x, d.y);
}

// barrier of one group's warps (named barrier 1 + group)
template <int GW>
__device__ __forceinline__ void group_sync(int grp) {
  if constexpr (GW == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + grp), "n"(32 * GW) : "memory");
}

// split operand step k of an array of KP k16 steps (hi words of 32 lanes, then
// lo words) followed by the k8 step (hi, hi, lo, lo)
__device__ __forceinline__ Frag get_frag(const uint4 *a, int k, int lane) {
  const uint4 h = a[k * 64 + lane], l = a[k * 64 + 32 + lane];
  return Frag{{h.x, h.y, h.z, h.w}, {l.x, l.y, l.z, l.w}};
}
__device__ __forceinline__ void put_frag(uint4 *a, int k, int lane, const Frag &f) {
  a[k * 64 + lane] = make_uint4(f.h[0], f.h[1], f.h[2], f.h[3]);
  a[k * 64 + 32 + lane] = make_uint4(f.l[0], f.l[1], f.l[2], f.l[3]);
}
__device__ __forceinline__ Frag8 get_frag8(const uint4 *a, int KP, int lane) {
  const uint4 q = a[KP * 64 + lane];
  return Frag8{{q.x, q.y}, {q.z, q.w}};
}
__device__ __forceinline__ void put_frag8(uint4 *a, int KP, int lane, const Frag8 &f) {
  a[KP * 64 + lane] = make_uint4(f.h[0], f.h[1], f.l[0], f.l[1]);
}

// sources of the tile's elements k0 .. k0 + 15, in the reference's place: added
// to the projected rhs_p (acous_elas_cpp/okl/ElasKernelsWADG.okl:400-403).
// add(row in the tile, amplitude, vector)
template <class F>
__device__ __forceinline__ void tile_sources(const WarpParams &P, int Np, int shot, int k0, F &&add) {
  const int tb = shot * P.nt32 + k0 / 32, te = shot * P.nt32 + min(k0 + 15, P.K - 1) / 32;
  const int j0 = __ldg(P.src_tile + tb), j1 = __ldg(P.src_tile + te + 1);
  if (j1 <= j0) return;
  const float amp = warp_ricker((float)(*P.time) + P.cstage * P.fdt, P.f0, P.tR, P.samp);
  for (int s = j0; s < j1; ++s) {
    const int e = __ldg(P.src_elem + s) - k0;
    if (e >= 0 && e < 16) add(e, amp, P.src_vec + (size_t)s * Np);
  }
}

// launch parameters common to both forms; the grid walks nit items
inline WarpParams warp_params(const WarpPlan &pl, const float *Qin, float *Qout, float *res, float fa,
                              float fb, float fdt, float cstage) {
  WarpParams P{};
  P.K = pl.K, P.K0 = pl.K0, P.Kc = pl.Kc > 0 ? pl.Kc : pl.K, P.Nq = pl.Nq, P.bc = pl.bc;
  P.pat_off = pl.pat_off, P.table_ints = pl.table_ints, P.nt32 = (pl.K + 31) / 32;
  P.Nq16 = (pl.Nq + 15) / 16 * 16;
  P.oDt = pl.oDt, P.oL = pl.oL, P.oLt = pl.oLt, P.oV = pl.oV, P.oVt = pl.oVt, P.oP = pl.oP;
  P.oM = pl.oM;
  P.ops_n = pl.ops_n;
  P.fa = fa, P.fb = fb, P.fdt = fdt, P.cstage = cstage;
  P.iD = pl.iD, P.iL = pl.iL, P.iV = pl.iV, P.iP = pl.iP, P.vnorm = pl.vnorm;
  P.Qin = Qin, P.Qout = Qout, P.res = res;
  P.geo = pl.geo, P.c2p = pl.c2p, P.c2max = pl.c2max, P.nbr = pl.nbr;
  P.tables = pl.tables, P.ops = pl.ops;
  P.src_tile = pl.src_tile, P.src_elem = pl.src_elem, P.src_vec = pl.src_vec;
  P.f0 = pl.f0, P.tR = pl.tR, P.samp = pl.samp, P.time = pl.time;
  P.ntile = (P.Kc - P.K0 + 15) / 16;
  P.nit = P.ntile * pl.S;
  return P;
}

// items walked by `per_cta` workers (warps or groups) of each CTA; returns the grid
inline int warp_grid(const WarpPlan &pl, int per_cta, WarpParams &P) {
  const int ctas = pl.max_ctas > 0 && pl.max_ctas < pl.nsm ? pl.max_ctas : pl.nsm;
  int grid = ctas;
  if (P.nit <= ctas * per_cta) {
    // at most one item per worker: spread the items over the SMs first
    grid = P.nit < ctas ? P.nit : ctas;
    P.bs = 1, P.ws = grid;
  } else {
    // a CTA's workers walk neighbouring tiles, whose traces they share in L1
    P.bs = per_cta, P.ws = 1;
  }
  P.step_shot = grid * per_cta / P.ntile, P.step_tile = grid * per_cta % P.ntile;
  return grid;
}

}  // namespace bbw
