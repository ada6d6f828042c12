// efie_far_pair_beta (far_df.h) with the trial points two by two in packed FP32 (pack2.h): the double-float
// part of a point pair is 150 of its 180 FP32 instructions, and the kernel's issue slots are what bounds it.
// Lane for lane the operations and their roundings are those of dfloat.h; only the running sum of the
// beta term is split into the even and the odd trial points.  The FP32 moments of the alpha term are
// summed point by point in the order of efie_far_pair_beta.  (device only)
#pragma once
#include "far_df.h"
#include "pack2.h"

namespace dfl {

using pk::f2;
struct df2 {
  f2 hi, lo;
};
__device__ __forceinline__ df2 both(df a) { return {pk::both(a.hi), pk::both(a.lo)}; }
__device__ __forceinline__ df2 two_sum(f2 a, f2 b) {
  const f2 s = pk::add(a, b), bb = pk::sub(s, a);
  return {s, pk::add(pk::sub(a, pk::sub(s, bb)), pk::sub(b, bb))};
}
__device__ __forceinline__ df2 two_diff(f2 a, f2 b) {  // two_sum(a, -b)
  const f2 s = pk::sub(a, b), bb = pk::sub(s, a);
  return {s, pk::sub(pk::sub(a, pk::sub(s, bb)), pk::add(b, bb))};
}
// a b - p (a single instruction takes the sign along, the packed one does not)
__device__ __forceinline__ f2 prod_rest(f2 a, f2 b, f2 p) {
  return pk::make(fmaf(pk::lo(a), pk::lo(b), -pk::lo(p)), fmaf(pk::hi(a), pk::hi(b), -pk::hi(p)));
}
__device__ __forceinline__ df2 mulu(df2 a, df2 b) {
  const f2 p = pk::mul(a.hi, b.hi);
  return {p, pk::fma(a.hi, b.lo, pk::fma(a.lo, b.hi, prod_rest(a.hi, b.hi, p)))};
}
__device__ __forceinline__ void acc(df2& a, df2 x) {
  const df2 s = two_sum(a.hi, x.hi);
  a.hi = s.hi;
  a.lo = pk::add(a.lo, pk::add(s.lo, x.lo));
}
__device__ __forceinline__ df2 addu(df2 a, df2 b) {
  const df2 s = two_sum(a.hi, b.hi);
  return {s.hi, pk::add(s.lo, pk::add(a.lo, b.lo))};
}
__device__ __forceinline__ df2 subu(df2 a, df2 b) {
  const df2 s = two_diff(a.hi, b.hi);
  return {s.hi, pk::add(s.lo, pk::sub(a.lo, b.lo))};
}
__device__ __forceinline__ df2 rsqrtu(df2 a) {
  const f2 y0 = pk::make(rsqrtf(pk::lo(a.hi)), rsqrtf(pk::hi(a.hi)));
  const f2 p = pk::mul(y0, y0);
  const df2 ay2 = mulu(a, df2{p, prod_rest(y0, y0, p)});
  const f2 e = pk::sub(pk::sub(pk::both(1.f), ay2.hi), ay2.lo);
  return {y0, pk::mul(pk::mul(y0, e), pk::both(0.5f))};
}
// sine and cosine of th, |th| < 2^15, left unnormalised: th = n pi/256 + t from a table of 512 points (tab[4][512]:
// sin hi, lo, cos hi, lo), so that t^2/2 < 2e-5 and everything but the table value and its product with t
// is FP32: 44 instructions per angle for the 76 of 64 points.  Absolute error below 4e-12.
__device__ __forceinline__ void sincos_tab2(df2 th, const float* tab, df2* s, df2* c) {
  const f2 f = pk::fma(th.hi, pk::both(81.4873275756836f), pk::both(12582912.f));  // 256 / pi, nearest whole number
  const f2 n = pk::sub(f, pk::both(12582912.f));
  const f2 np = pk::mul(n, pk::both(-0.012271846644580364f));
  const f2 t = pk::add(th.hi, np);  // exact; the rest below: 2^-24 of th
  f2 e = pk::sub(th.lo, pk::fma(n, pk::both(0.012271846644580364f), np));
  e = pk::fma(n, pk::both(3.4149522099014007e-10f), e);
  e = pk::fma(n, pk::both(1.3399410234420952e-17f), e);
  const float* e0 = tab + (__float_as_uint(pk::lo(f)) & 511u);
  const float* e1 = tab + (__float_as_uint(pk::hi(f)) & 511u);
  const f2 sh = pk::make(e0[0], e1[0]), sl = pk::make(e0[512], e1[512]), ch = pk::make(e0[1024], e1[1024]),
           cl = pk::make(e0[1536], e1[1536]);
  const f2 tt = pk::add(t, e), t2 = pk::mul(tt, tt);
  const f2 c1 = pk::mul(t2, pk::fma(t2, pk::both(1.f / 24.f), pk::both(-0.5f)));      // cos t - 1
  const f2 e3 = pk::fma(pk::mul(tt, t2), pk::both(-1.f / 6.f), e);                    // sin t - t.hi
  // sin (table + t) = sh + ch t + (sl + cl t + ch e3 + sh c1)
  // and cos (table + t) = ch - sh t + (cl + ch c1 - (sl t + sh e3))
  const f2 p = pk::mul(ch, t), q = pk::mul(sh, t);
  const df2 us = two_sum(sh, p), uc = two_diff(ch, q);
  const f2 v = pk::fma(ch, e3, pk::fma(cl, t, prod_rest(ch, t, p))), w = pk::fma(sh, e3, pk::fma(sl, t, prod_rest(sh, t, q)));
  *s = {us.hi, pk::add(us.lo, pk::add(pk::fma(sh, c1, sl), v))};
  *c = {uc.hi, pk::add(uc.lo, pk::sub(pk::fma(ch, c1, cl), w))};
}

// a trial cell's points in pairs: (b, b + 1) of each component's high and low parts, |eta|^2, and the high
// parts (eta rounded to FP32) doubled for the complex moments
template <int NI>
struct EtaPairs {
  float2 hi[NI / 2][3], lo[NI / 2][3], s_hi[NI / 2], s_lo[NI / 2];
  float2 dup[NI][3];
};
__device__ __forceinline__ f2 ld(const float2& x) { return f2{x}; }

// wab[a][b / 2]: high parts of (b, b + 1), low parts
template <int NO, int NI>
__device__ __forceinline__ void efie_far_pair_beta2(const df* d, const df (*tau)[3], const df (*sig)[3], const df (*xi)[3],
                                                    const float4 (*wab)[NI / 2], const EtaPairs<NI>& E, df k, cdf alpha,
                                                    cdf beta, const float* tab, cdf* out) {
  const f2 z0 = pk::both(0.f);
  df2 Mr{z0, z0}, Mi{z0, z0};
  cf M1 = cf{0.f, 0.f};
  f2 V1[3], V2[3];
  for (int c = 0; c < 3; ++c) V1[c] = V2[c] = z0;
  const df2 kk = both(k);
#pragma unroll 1
  for (int a = 0; a < NO; ++a) {
    df dx[3];
    float xf[3];
    df2 dx2[3];
    for (int c = 0; c < 3; ++c) {
      dx[c] = adds(d[c], xi[a][c]);
      xf[c] = f32(xi[a][c]);
      dx2[c] = both(dx[c]);
    }
    const df2 A = both(dot3u(dx, dx));
    f2 U0 = z0;
#pragma unroll 1
    for (int b = 0; b < NI / 2; ++b) {
      f2 eh[3];
      for (int c = 0; c < 3; ++c) eh[c] = ld(E.hi[b][c]);
      df2 Pd = mulu(dx2[0], df2{eh[0], ld(E.lo[b][0])});
      acc(Pd, mulu(dx2[1], df2{eh[1], ld(E.lo[b][1])}));
      acc(Pd, mulu(dx2[2], df2{eh[2], ld(E.lo[b][2])}));
      df2 R2 = A;
      acc(R2, df2{ld(E.s_hi[b]), ld(E.s_lo[b])});
      const f2 m2 = pk::both(-2.f);
      acc(R2, df2{pk::mul(Pd.hi, m2), pk::mul(Pd.lo, m2)});
      const df2 iR = rsqrtu(R2);
      const df2 R = mulu(R2, iR);
      df2 sn, cs;
      sincos_tab2(mulu(kk, R), tab, &sn, &cs);
      const float4 w = wab[a][b];
      const df2 amp = mulu(iR, df2{pk::make(w.x, w.y), pk::make(w.z, w.w)});
      const df2 kr = mulu(amp, cs), ki = mulu(amp, sn);  // (K's imaginary part is -ki)
      acc(Mr, kr);
      acc(Mi, ki);
      const f2 p = pk::fma(pk::both(xf[0]), eh[0], pk::fma(pk::both(xf[1]), eh[1], pk::mul(pk::both(xf[2]), eh[2])));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float x = h ? add_rn(pk::hi(kr.hi), pk::hi(kr.lo)) : add_rn(pk::lo(kr.hi), pk::lo(kr.lo));
        const float y = h ? add_rn(-pk::hi(ki.hi), -pk::hi(ki.lo)) : add_rn(-pk::lo(ki.hi), -pk::lo(ki.lo));
        const f2 K = pk::make(x, y);
        U0 = pk::add(U0, K);
        const float ph = h ? pk::hi(p) : pk::lo(p);
        M1.x = fmaf(x, ph, M1.x);
        M1.y = fmaf(y, ph, M1.y);
        for (int c = 0; c < 3; ++c) V2[c] = pk::fma(K, ld(E.dup[2 * b + h][c]), V2[c]);
      }
    }
    for (int c = 0; c < 3; ++c) V1[c] = pk::fma(U0, pk::both(xf[c]), V1[c]);
  }
  const df mr = add(df{pk::lo(Mr.hi), pk::lo(Mr.lo)}, df{pk::hi(Mr.hi), pk::hi(Mr.lo)});
  const df mi = add(df{pk::lo(Mi.hi), pk::lo(Mi.lo)}, df{pk::hi(Mi.hi), pk::hi(Mi.lo)});
  cf v1[3], v2[3];
  for (int c = 0; c < 3; ++c) {
    v1[c] = cf{pk::lo(V1[c]), pk::hi(V1[c])};
    v2[c] = cf{pk::lo(V2[c]), pk::hi(V2[c])};
  }
  efie_beta_block(cdf{mr, neg(mi)}, M1, v1, v2, tau, sig, alpha, beta, out);
}

}  // namespace dfl
