// Float64 interpolation on the integer pipe.
//
// The float64 pipe of this GPU issues 2 lanes per SM and clock (measured:
// fma, add, compare and every float64 conversion 1.7-2.0), the 32 x 32 -> 64
// multiply-add (IMAD.WIDE) 32.  A tricubic query is ~170 (scalar) to ~530
// ('both') float64 operations, so the float64 evaluators were bound by that
// pipe at 85-250 clocks per query and SM.  Here the same contraction runs in
// 61-bit block fixed point: the samples of one 4^dim block (or of one staged
// tile) share the exponent of their largest, weights are 62-bit fractions, a
// product of two such numbers is three IMAD.WIDE, and every result is rounded
// to float64 once.
//
// Accuracy.  A sample is exact down to 2^-8 of the largest (53-bit significand
// in 61 bits) and otherwise cut at 2^-61 of it; a product drops its low x low
// word and the stages round at 2^-60 of the largest sample.  Against quadruple
// precision, random queries: 1.1e-16 of the block's largest sample with the final
// rounding, 8.1e-16 for float64 arithmetic.  Both errors scale with samples, but not
// with the same ones: float64 arithmetic weights each rounding with its sample's
// weight, the cut here is one for the block.  So where the samples that count are
// far below the largest (by 2^8 and more) and the weights of the large ones vanish,
// float64 arithmetic keeps bits that the cut takes.  On grid points, where it loses
// nothing at all, the samples are taken themselves (at_node in eval.cuh); close to
// one, or on a grid line or plane through small samples beside large ones, a result
// has an absolute error of 0.02 (3D) to 0.04 (4D) of 2^-53 of the largest sample (of
// the footprint in a staged bin; eight times that of the cell's largest corner
// where that sets the scale) and no relative one.
//
// Words: a number is h 2^32 + l with l a signed word, so that the split of a
// 64-bit value into words is its two registers but for one carry.
#pragma once

#include "arb_common.cuh"

namespace arb {

constexpr int FX_DB = 61;                    // |sample| < 2^FX_DB
constexpr int FX_EMIN = 64, FX_EMAX = 2040;  // biased exponents of the largest sample that the scaling holds

// One weight of an axis and its derivative weight.
struct FxWord {
  int wh, wl, dh, dl;
};

template <typename T>
__host__ __device__ __forceinline__ T fx_sel(const T v[4], int k) {
  return k == 0 ? v[0] : (k == 1 ? v[1] : (k == 2 ? v[2] : v[3]));
}

struct FxW {  // one axis: weights w and derivative weights d (times 2^-DS), times 2^62, as words
  int wh[4], wl[4], dh[4], dl[4];
  __host__ __device__ __forceinline__ FxWord get(int, int k) const {
    return FxWord{fx_sel(wh, k), fx_sel(wl, k), fx_sel(dh, k), fx_sel(dl, k)};
  }
};

// acc + a b: one IMAD.WIDE.  In PTX, because a product of words that come from
// shifts of 64-bit values is otherwise compiled as a 64 x 64-bit one; as a
// product and a sum, which the assembler fuses (mad.wide.s32 takes one more
// instruction: 26 against 14 for 12 of them).
__host__ __device__ __forceinline__ long long fx_mad(int a, int b, long long acc) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("{\n\t.reg .s64 p;\n\tmul.wide.s32 p, %1, %2;\n\tadd.s64 %0, p, %3;\n\t}" : "=l"(r) : "r"(a), "r"(b), "l"(acc));
  return r;
#else
  return (long long)a * b + acc;
#endif
}

__host__ __device__ __forceinline__ void fx_split(long long v, int &h, int &l) {
  h = (int)((v + 0x80000000LL) >> 32);
  l = (int)(unsigned)v;
}

// Sum of products, times 2^(S - 64): hh holds the high x high products, cr the
// mixed ones (in units of 2^32 less); low x low products are dropped.  The
// start values round cr and carry the split's 2^31.  Bounds, with |a| < 1.25 2^61
// and sums of |weights| <= 1.25 2^62 (1.5 2^62 with |a| < 2^61): |cr| < 2^63.
template <int S>
struct FxAcc {
  long long hh, cr;
  __host__ __device__ __forceinline__ FxAcc() : hh(1LL << (31 - S)), cr(1LL << (31 - S)) {}
  __host__ __device__ __forceinline__ void mac(int ah, int al, int bh, int bl) {
    hh = fx_mad(ah, bh, hh);
    cr = fx_mad(ah, bl, cr);
    cr = fx_mad(al, bh, cr);
  }
  __host__ __device__ __forceinline__ long long sum() const { return hh * (1 << S) + (cr >> (32 - S)); }
  __host__ __device__ __forceinline__ void norm(int &h, int &l) const {
    const long long v = sum();
    h = (int)(v >> 32);
    l = (int)((unsigned)v ^ 0x80000000u);
  }
  __host__ __device__ __forceinline__ long long value() const { return sum() - 0x80000000LL; }
};

// x >> s for 0 <= s < 2^16; 0 from 64 on (the hardware shift clamps).
__host__ __device__ __forceinline__ unsigned long long fx_shr(unsigned long long x, int s) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
#else
  return s > 63 ? 0ULL : x >> s;
#endif
}

__host__ __device__ __forceinline__ int fx_clz(unsigned long long x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// Significand of a float64 (its implicit one assumed) with the leading one in bit 62.
__host__ __device__ __forceinline__ unsigned long long fx_significand(unsigned long long b) {
  return ((b << 10) & 0x7fffffffffffffffULL) | 0x4000000000000000ULL;
}

// Float64 bits b, in units of 2^(emax - 1022 - FX_DB), as words.  Zeros and
// subnormals (exponent 0) shift out to 0 (emax >= FX_EMIN).
__host__ __device__ __forceinline__ void fx_sample(unsigned long long b, int emax, int &h, int &l) {
  const int e = (int)(b >> 52) & 0x7ff;
  const long long x = (long long)fx_shr(fx_significand(b), 63 - FX_DB + emax - e);
  const long long s = (long long)b >> 63;
  fx_split((x ^ s) - s, h, l);
}

// R 2^(ex - 1022 - FX_DB) rounded to nearest even as float64 (ex within the
// scaling's range; |R| < 2^63).
__host__ __device__ __forceinline__ unsigned long long fx_to_double_bits(long long R, int ex) {
  const long long sg = R >> 63;
  const unsigned long long m0 = (unsigned long long)((R ^ sg) - sg);
  const int z = fx_clz(m0 | 1ULL);
  const unsigned long long a = m0 << z;  // leading one in bit 63
  // to 53 bits: half less one, plus the last kept bit (to even)
  const unsigned long long m = (a + 0x3ffULL + ((a >> 11) & 1ULL)) >> 11;
  const unsigned long long c = a + 0x3ffULL + ((a >> 11) & 1ULL) < a ? 1ULL << 53 : 0ULL;  // carry out of bit 63
  const unsigned long long bits = ((unsigned long long)(unsigned)(ex + 63 - FX_DB - z) << 52) + (m | c);
  return m0 ? bits | ((unsigned long long)sg & 0x8000000000000000ULL) : 0ULL;  // m carries its leading one
}

__device__ __forceinline__ double fx_to_double(long long R, int ex) {
  return __longlong_as_double((long long)fx_to_double_bits(R, ex));
}

// Catmull-Rom weights and derivative weights of the fraction t (float64
// bits, 0 <= t < 1).  T = t 2^61, T2 = t^2 2^61, T3 = t^3 2^61:
//   w0 2^62 = -T + 2 T2 - T3, w2 2^62 = T + 4 T2 - 3 T3, w3 2^62 = T3 - T2, w1 = 1 - (the others);
//   d0 2^62 = -2^61 + 4 T - 3 T2, d2 2^62 = 2^61 + 8 T - 9 T2, d3 2^62 = 3 T2 - 2 T, d1 = -(the others).
// The sums 1 and 0 hold exactly, so errors of T2 and T3 act on differences of
// samples only.  DS: derivative weights are stored times 2^-DS, for FxAcc's bounds
// (absolute sums: w 1.25, d 3 2^-DS).
template <int DS>
__host__ __device__ __forceinline__ void fx_axis(unsigned long long tbits, FxW &o) {
  using u64 = unsigned long long;
  const int e = (int)(tbits >> 52) & 0x7ff;
  const u64 T = fx_shr(fx_significand(tbits), 1024 - e);
  int th, tl, sh, sl;
  fx_split((long long)T, th, tl);
  const u64 T2 = ((u64)fx_mad(th, th, 0) << 3) + (u64)(fx_mad(th, tl, 1LL << 27) >> 28);
  fx_split((long long)T2, sh, sl);
  const u64 T3 = ((u64)fx_mad(th, sh, 0) << 3) + (u64)(fx_mad(th, sl, fx_mad(tl, sh, 1LL << 28)) >> 29);
  const u64 one = 1ULL << 62, half = 1ULL << 61, rnd = 1ULL << (DS - 1);
  const u64 w0 = 2 * T2 - T - T3, w2 = T + 4 * T2 - 3 * T3, w3 = T3 - T2;
  fx_split((long long)w0, o.wh[0], o.wl[0]);
  fx_split((long long)(one - w0 - w2 - w3), o.wh[1], o.wl[1]);
  fx_split((long long)w2, o.wh[2], o.wl[2]);
  fx_split((long long)w3, o.wh[3], o.wl[3]);
  // modulo 2^64 on the way, within 1.4 2^62 at the end
  const long long d0 = (long long)(4 * T - 3 * T2 - half + rnd) >> DS;
  const long long d2 = (long long)(half + 8 * T - 9 * T2 + rnd) >> DS;
  const long long d3 = (long long)(3 * T2 - 2 * T + rnd) >> DS;
  fx_split(d0, o.dh[0], o.dl[0]);
  fx_split(-(d0 + d2 + d3), o.dh[1], o.dl[1]);
  fx_split(d2, o.dh[2], o.dl[2]);
  fx_split(d3, o.dh[3], o.dl[3]);
}

#ifdef __CUDACC__
// Weights of outer axes (4D: z and t; z of the 3D tiles with a gradient) in shared memory, a
// column a thread: in registers they were 32 of the ~190 that fx_eval4 has alive, and the
// loops over k and t picked from them by selects (1.5e6 scalar queries on 33 x 41
// x 29 x 17, one lane a query: 1122 -> 1049 us).  Kernels that use them have at
// most FX_ZT_THREADS threads.
constexpr int FX_ZT_THREADS = 128;
template <int AXES>
struct FxZTCols {
  static __device__ __forceinline__ int4 *column() {
    __shared__ int4 zt[4 * AXES * FX_ZT_THREADS];
    return zt + threadIdx.x;
  }
  static __device__ __forceinline__ void set(int axis, const FxW &w) {
#pragma unroll
    for (int k = 0; k < 4; ++k) column()[(4 * axis + k) * FX_ZT_THREADS] = make_int4(w.wh[k], w.wl[k], w.dh[k], w.dl[k]);
  }
  __device__ __forceinline__ FxWord get(int axis, int k) const {
    const int4 v = column()[(4 * axis + k) * FX_ZT_THREADS];
    return FxWord{v.x, v.y, v.z, v.w};
  }
};
using FxZT = FxZTCols<2>;  // 4D: z, t
using FxZ = FxZTCols<1>;   // 3D: z
#endif

// Tricubic contraction of a 4x4x4 block of F fields: R[f] the values and (F
// != 3) G[a] the last field's derivatives times 2^-1, in the fields' units.
// SRC::point(i, j, k, h, l) gives the words of a block point's fields.
// Planes run in a rolled loop: unrolled, the body is four times as long and
// the kernel waits on instruction fetch.  A sum of four products is a chain of
// 8 dependent IMAD.WIDE, and at three warps per scheduler the chains have to
// hide each other's latency: the sums of RB rows and all fields advance
// together, point by point.
template <int F, class SRC, class WY, class WZ>
__host__ __device__ __forceinline__ void fx_eval3(const SRC &src, const FxW &wx, const WY &wy, const WZ &wz,
                                                  long long R[F], long long G[3]) {
  constexpr bool GRAD = F != 3;
  constexpr int RB = F == 4 ? 1 : (F == 3 ? 2 : 4);
  FxAcc<3> V[F], gx, gy, gz;
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    FxAcc<2> Y[F], yx, yy;
#pragma unroll
    for (int jb = 0; jb < 4; jb += RB) {
      FxAcc<1> a[RB][F], d[RB];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          int h[F], l[F];
          src.point(i, jb + r, k, h, l);
#pragma unroll
          for (int f = 0; f < F; ++f) a[r][f].mac(h[f], l[f], wx.wh[i], wx.wl[i]);
          if (GRAD) d[r].mac(h[F - 1], l[F - 1], wx.dh[i], wx.dl[i]);
        }
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const FxWord v = wy.get(0, jb + r);
        int h = 0, l = 0;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          a[r][f].norm(h, l);
          Y[f].mac(h, l, v.wh, v.wl);
        }
        if (GRAD) {
          yy.mac(h, l, v.dh, v.dl);
          d[r].norm(h, l);
          yx.mac(h, l, v.wh, v.wl);
        }
      }
    }
    const FxWord u = wz.get(0, k);
    int h = 0, l = 0;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      Y[f].norm(h, l);
      V[f].mac(h, l, u.wh, u.wl);
    }
    if (GRAD) {
      gz.mac(h, l, u.dh, u.dl);
      yx.norm(h, l);
      gx.mac(h, l, u.wh, u.wl);
      yy.norm(h, l);
      gy.mac(h, l, u.wh, u.wl);
    }
  }
#pragma unroll
  for (int f = 0; f < F; ++f) R[f] = V[f].value();
  if (GRAD) {
    G[0] = gx.value();
    G[1] = gy.value();
    G[2] = gz.value();
  }
}

// Quadcubic contraction of a 4^4 block of one field: the 4-fold Catmull-Rom
// sum plus sum_c T_c prod_a b_{c_a}(x_a), T_c = S_{c-1} - S_c, with S_c the
// (1/16) mixed fourth differences and b the slope-Hermite basis (see
// eval_otf4).  b_0 = -2 w0 and b_1 = 2 w3, so the factors 2^4 cancel the 1/16
// and the correction uses the same weights; the differences are exact
// integers, kept 2^-5 down so that T_c fits (the correction's weights are at
// most 0.074^4, its derivatives' 0.5 0.074^3).  Derivative weights are stored
// times 2^-2 (DS = 2).  GRADF: also the derivatives (times 2^-2) into G.
// SRC::UNROLL: planes of a slab unrolled (words from a tile) or in a loop (with
// the conversions of a gathered block the body would outgrow the instruction
// cache).
template <bool GRADF, class SRC, class ZT>
__host__ __device__ __forceinline__ void fx_eval4(const SRC &src, const FxW w[2], const ZT &zt, long long &R,
                                                  long long G[4]) {
  FxAcc<3> V, gt;
  FxAcc<2> gx, gy, gz;
  long long S[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) S[m] = 0;
#pragma unroll 1
  for (int t = 0; t < 4; ++t) {
    FxAcc<2> Z, zx, zy;
    FxAcc<3> zz;
    long long E2[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) E2[m] = 0;
#pragma unroll SRC::UNROLL
    for (int k = 0; k < 4; ++k) {
      FxAcc<2> Y, yx;
      FxAcc<3> yy;
      FxAcc<1> a[4];
      FxAcc<2> d[4];
      // words of the x, y differences of corner (m & 1, m >> 1): sums of four
      // samples, the low words 2^-3 down so that they fit
      int eh[4], el[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          int h, l;
          src.point(i, j, k, t, &h, &l);
          a[j].mac(h, l, w[0].wh[i], w[0].wl[i]);
          if (GRADF) d[j].mac(h, l, w[0].dh[i], w[0].dl[i]);
          const int m = (i & 1) + 2 * (j & 1);
          const bool plus = (i >= 2) == (j >= 2);  // both in the upper or both in the lower half of the difference
          eh[m] = i < 2 && j < 2 ? h : (plus ? eh[m] + h : eh[m] - h);
          el[m] = i < 2 && j < 2 ? l >> 3 : (plus ? el[m] + (l >> 3) : el[m] - (l >> 3));
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int h, l;
        a[j].norm(h, l);
        Y.mac(h, l, w[1].wh[j], w[1].wl[j]);
        if (GRADF) {
          yy.mac(h, l, w[1].dh[j], w[1].dl[j]);
          d[j].norm(h, l);
          yx.mac(h, l, w[1].wh[j], w[1].wl[j]);
        }
      }
      const FxWord wz = zt.get(0, k);
      int h, l;
      Y.norm(h, l);
      Z.mac(h, l, wz.wh, wz.wl);
      if (GRADF) {
        zz.mac(h, l, wz.dh, wz.dl);
        yx.norm(h, l);
        zx.mac(h, l, wz.wh, wz.wl);
        yy.norm(h, l);
        zy.mac(h, l, wz.wh, wz.wl);
      }
      const long long up = k >= 2 ? 0 : -1, even = (k & 1) - 1;
#pragma unroll
      for (int m = 0; m < 4; ++m) {  // times 2^-5
        const long long e = (long long)((unsigned long long)(long long)eh[m] << 27) + (el[m] >> 2);
        const long long v = (e ^ up) - up;
        E2[m] += v & even;
        E2[m + 4] += v & ~even;
      }
    }
    const FxWord wt = zt.get(1, t);
    int h, l;
    Z.norm(h, l);
    V.mac(h, l, wt.wh, wt.wl);
    if (GRADF) {
      gt.mac(h, l, wt.dh, wt.dl);
      zx.norm(h, l);
      gx.mac(h, l, wt.wh, wt.wl);
      zy.norm(h, l);
      gy.mac(h, l, wt.wh, wt.wl);
      zz.norm(h, l);
      gz.mac(h, l, wt.wh, wt.wl);
    }
    const long long up = t >= 2 ? 0 : -1, even = (t & 1) - 1;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const long long v = (E2[m] ^ up) - up;
      S[m] += v & even;
      S[m + 8] += v & ~even;
    }
  }
  // correction: contract T_c (units 2^5) with (-w0, w3) along x, y, z, t; with
  // GRADF one product more per derivative.  The weights are at most 0.074 (0.5
  // for a derivative), so the factor 2^5 comes back as 2^2 after x, 2^2 after y and 2 at the end.
  long long Tc[16];
  Tc[0] = -S[0];
#pragma unroll
  for (int m = 1; m < 16; ++m) Tc[m] = S[m - 1] - S[m];
  int Ch[8], Cl[8], Dh[8], Dl[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    int h0, l0, h1, l1;
    fx_split(-Tc[2 * m], h0, l0);
    fx_split(Tc[2 * m + 1], h1, l1);
    FxAcc<4> a, d;
    a.mac(h0, l0, w[0].wh[0], w[0].wl[0]);
    a.mac(h1, l1, w[0].wh[3], w[0].wl[3]);
    a.norm(Ch[m], Cl[m]);
    if (GRADF) {
      d.mac(h0, l0, w[0].dh[0], w[0].dl[0]);
      d.mac(h1, l1, w[0].dh[3], w[0].dl[3]);
      d.norm(Dh[m], Dl[m]);
    }
  }
  int Yh[4], Yl[4], Xh[4], Xl[4], Gh[4], Gl[4];  // value, d/dx, d/dy along y
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    FxAcc<4> a, d, e;
    a.mac(-Ch[2 * m], -Cl[2 * m], w[1].wh[0], w[1].wl[0]);
    a.mac(Ch[2 * m + 1], Cl[2 * m + 1], w[1].wh[3], w[1].wl[3]);
    a.norm(Yh[m], Yl[m]);
    if (GRADF) {
      d.mac(-Dh[2 * m], -Dl[2 * m], w[1].wh[0], w[1].wl[0]);
      d.mac(Dh[2 * m + 1], Dl[2 * m + 1], w[1].wh[3], w[1].wl[3]);
      d.norm(Xh[m], Xl[m]);
      e.mac(-Ch[2 * m], -Cl[2 * m], w[1].dh[0], w[1].dl[0]);
      e.mac(Ch[2 * m + 1], Cl[2 * m + 1], w[1].dh[3], w[1].dl[3]);
      e.norm(Gh[m], Gl[m]);
    }
  }
  FxAcc<3> c0, cx, cy, cz, ct;
  const FxWord z0 = zt.get(0, 0), z3 = zt.get(0, 3);
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    FxAcc<2> a, b, c, d;
    int h, l;
    const int sg = m ? 1 : -1;
    const FxWord u = zt.get(1, m ? 3 : 0);
    a.mac(-Yh[2 * m], -Yl[2 * m], z0.wh, z0.wl);
    a.mac(Yh[2 * m + 1], Yl[2 * m + 1], z3.wh, z3.wl);
    a.norm(h, l);
    c0.mac(sg * h, sg * l, u.wh, u.wl);
    if (GRADF) {
      ct.mac(sg * h, sg * l, u.dh, u.dl);
      b.mac(-Xh[2 * m], -Xl[2 * m], z0.wh, z0.wl);
      b.mac(Xh[2 * m + 1], Xl[2 * m + 1], z3.wh, z3.wl);
      b.norm(h, l);
      cx.mac(sg * h, sg * l, u.wh, u.wl);
      c.mac(-Gh[2 * m], -Gl[2 * m], z0.wh, z0.wl);
      c.mac(Gh[2 * m + 1], Gl[2 * m + 1], z3.wh, z3.wl);
      c.norm(h, l);
      cy.mac(sg * h, sg * l, u.wh, u.wl);
      d.mac(-Yh[2 * m], -Yl[2 * m], z0.dh, z0.dl);
      d.mac(Yh[2 * m + 1], Yl[2 * m + 1], z3.dh, z3.dl);
      d.norm(h, l);
      cz.mac(sg * h, sg * l, u.wh, u.wl);
    }
  }
  R = V.value() + c0.value();
  if (GRADF) {
    G[0] = gx.value() + cx.value();
    G[1] = gy.value() + cy.value();
    G[2] = gz.value() + cz.value();
    G[3] = gt.value() + ct.value();
  }
}

// ---- blocks of the float64 grid ------------------------------------------------
// F fields of one point from p (F = 4: 16-byte loads), as words lo, hi.
template <int F>
__device__ __forceinline__ void fx_read(const double *p, uint32_t lo[F], uint32_t hi[F]) {
  if constexpr (F == 4) {
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p)), b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
    lo[0] = a.x;
    hi[0] = a.y;
    lo[1] = a.z;
    hi[1] = a.w;
    lo[2] = b.x;
    hi[2] = b.y;
    lo[3] = b.z;
    hi[3] = b.w;
  } else {
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const uint2 a = __ldg(reinterpret_cast<const uint2 *>(p) + f);
      lo[f] = a.x;
      hi[f] = a.y;
    }
  }
}

__device__ __forceinline__ unsigned long long fx_pair(uint32_t lo, uint32_t hi) {
  return ((unsigned long long)hi << 32) | lo;
}

// A gather of one lane per query is bound by L1 (one wavefront per lane and
// load), so a block is read once: its scale is set from the 8 corners of the
// query's own cell with FX_HEAD bits of headroom, and a sample above that
// (fit() false) sends the query to scale(), which reads the whole block for
// its largest sample and no headroom.  The cut is then at 2^-58 of the cell's
// largest corner, still 2^5 below the float64 rounding of those samples.
// A field that is zero at all corners (one component of a planar field, the rest
// of a grid around a localised source) takes the lowest exponent, which no
// other block has here, and holds if the block has no other high word: its result
// is zero.  (Samples below 2^-1042, which set the low word alone, count as zeros.)
// Sent to scale() instead, one such component made every query read its block
// three times: 1e6 vector queries on 64^3 710 us, now 450, with float64
// arithmetic 670.
constexpr int FX_HEAD = 3;
__host__ __device__ __forceinline__ bool fx_fits(uint32_t over, int emax) {
  return emax < FX_EMIN + FX_HEAD ? over == 0 : (int)((over + 1) >> 20) <= emax;
}

// Largest sample of a set, by bits: the largest high word without its sign,
// and whether any low word is set (to tell zeros from subnormals).
struct FxMax {
  uint32_t m = 0, z = 0;
  __device__ __forceinline__ void add(uint32_t hi, uint32_t lo) {
    m = max(m, hi & 0x7fffffffu);
    z |= lo;
  }
  // Exponent for the scaling, one more for a sample that rounds up to the next
  // (then four high words add up in 32 bits); false where it does not apply
  // (infinities, NaN, magnitudes outside 2^[-959, 1017]).  All zeros: any.
  __device__ __forceinline__ bool exponent(int &e) const {
    e = (int)((m + 1) >> 20);
    if ((m | z) == 0) e = 1023;
    return e >= FX_EMIN && e <= FX_EMAX;
  }
  // The same for a cell's corners: with headroom, FX_EMIN for zeros.
  __device__ __forceinline__ bool corners(int &e) const {
    e = (int)((m + 1) >> 20);
    const bool ok = e >= FX_EMIN && e <= FX_EMAX - FX_HEAD;
    e += FX_HEAD;
    if ((m | z) == 0) e = FX_EMIN;
    return ok || (m | z) == 0;
  }
};

// STEP: doubles between points (F, or 4 for |B| of a 'both' grid alone).
template <int F, int STEP = F>
struct FxGrid3 {
  const double *p;  // block corner
  int64_t sy, sz;   // strides of y, z in doubles
  int emax[F];
  mutable uint32_t over[F];  // largest high word seen, per field
  __device__ __forceinline__ const double *at(int i, int j, int k) const { return p + i * STEP + j * sy + k * sz; }
  __device__ __forceinline__ void point(int i, int j, int k, int h[F], int l[F]) const {
    uint32_t lo[F], hi[F];
    fx_read<F>(at(i, j, k), lo, hi);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      over[f] = max(over[f], hi[f] & 0x7fffffffu);
      fx_sample(fx_pair(lo[f], hi[f]), emax[f], h[f], l[f]);
    }
  }
  __device__ __forceinline__ bool fit() const {
    bool ok = true;
#pragma unroll
    for (int f = 0; f < F; ++f) ok &= fx_fits(over[f], emax[f]);
    return ok;
  }
  // FULL: the whole block, exactly; otherwise the cell's corners, with headroom
  template <bool FULL>
  __device__ __forceinline__ bool scale() {
    constexpr int A = FULL ? 0 : 1, B = FULL ? 4 : 3;
    FxMax m[F];
#pragma unroll 1
    for (int k = A; k < B; ++k)
#pragma unroll
      for (int j = A; j < B; ++j)
#pragma unroll
        for (int i = A; i < B; ++i) {
          uint32_t lo[F], hi[F];
          fx_read<F>(at(i, j, k), lo, hi);
#pragma unroll
          for (int f = 0; f < F; ++f) m[f].add(hi[f], lo[f]);
        }
    bool ok = true;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      ok &= FULL ? m[f].exponent(emax[f]) : m[f].corners(emax[f]);
      over[f] = 0;
    }
    return ok;
  }
};

// One field of a 4D block; points lie `step` doubles apart along x.
struct FxGrid4 {
  static constexpr int UNROLL = 1;
  const double *p;
  int64_t step, sy, sz, st;
  int emax;
  mutable uint32_t over;  // largest high word seen
  __device__ __forceinline__ const double *at(int i, int j, int k, int t) const {
    return p + i * step + j * sy + k * sz + t * st;
  }
  __device__ __forceinline__ void point(int i, int j, int k, int t, int *h, int *l) const {
    uint32_t lo, hi;
    fx_read<1>(at(i, j, k, t), &lo, &hi);
    over = max(over, hi & 0x7fffffffu);
    fx_sample(fx_pair(lo, hi), emax, *h, *l);
  }
  __device__ __forceinline__ bool fit() const { return fx_fits(over, emax); }
  template <bool FULL>
  __device__ __forceinline__ bool scale() {
    constexpr int A = FULL ? 0 : 1, B = FULL ? 4 : 3;
    FxMax m;
#pragma unroll 1
    for (int t = A; t < B; ++t)
#pragma unroll 1
      for (int k = A; k < B; ++k)
#pragma unroll
        for (int j = A; j < B; ++j)
#pragma unroll
          for (int i = A; i < B; ++i) {
            uint32_t lo, hi;
            fx_read<1>(at(i, j, k, t), &lo, &hi);
            m.add(hi, lo);
          }
    over = 0;
    return FULL ? m.exponent(emax) : m.corners(emax);
  }
};

__device__ __forceinline__ unsigned long long fx_bits(double v) {
  return opaque_u64((unsigned long long)__double_as_longlong(v));
}

// Weights of a 4D block: x and y in registers, z and t in shared memory.
__device__ __forceinline__ void fx_weights4(const double frac[4], FxW w[2]) {
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    FxW v;
    fx_axis<2>(fx_bits(frac[a]), v);
    if (a < 2)
      w[a] = v;
    else
      FxZT::set(a - 2, v);
  }
}

// Values and gradient of a 3D block from its contraction (fx_eval3's units).
template <int F>
__device__ __forceinline__ void fx_finish3(const long long R[F], const long long G[3], const int emax[F],
                                           const double inv_h[4], double val[F], double grad[3]) {
#pragma unroll
  for (int f = 0; f < F; ++f) val[f] = fx_to_double(R[f], emax[f]);
  if (F != 3) {
#pragma unroll
    for (int a = 0; a < 3; ++a) grad[a] = fx_to_double(G[a], emax[F - 1] + 1) * inv_h[a];
  }
}

}  // namespace arb
