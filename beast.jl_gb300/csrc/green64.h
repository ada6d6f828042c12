// green64.h -- 1/R, R, cos(kR), sin(kR) from R^2 to FP64 accuracy with seven FP64 instructions.
//
// GB300 issues one FP64 instruction for about 60 FP32 or integer ones, so an FP64 kernel's time is
// its count of FP64 instructions, and CUDA's rsqrt and sincos take about 35 of them per value.  Here
// everything that is a small correction runs on the FP32 and integer pipes:
//   1/R   the FP32 reciprocal square root refined on float pairs (Newton, about 2^-45; the pairs'
//         error-free sums and products as in dfloat.h), then one FP64 Newton step;
//   kR    in steps of 2 pi / 4096: the FP64 product R (k 4096 / 2 pi), its integer and fractional
//         parts taken from the bits, the fraction as a float pair; the rounding of k 4096 / 2 pi is
//         made up for in FP32;
//   sin, cos   table value + correction: sin(a + t) = A + (B sin t + A (cos t - 1)) with A, B = sin,
//         cos of the table point (FP64, and as float pairs), |t| <= 7.7e-4; the parenthesis is at
//         most 7.7e-4, so pairs of floats (2^-47 relative) hold it to 2^-57, and one FP64 addition
//         finishes each.
// Accuracy: 1/R and R within 1 ulp; cos and sin within 2^-53 of the values at the rounded product
// (tests/test_green64.py).  Arguments kR below 64 steps (0.098; a table value's neighbourhood of 0
// would lose the relative accuracy of a small sine) or above 2^30 steps, and R^2 outside
// [2^-100, 2^90], take CUDA's functions in a call of their own.
// Host and device builds differ in the FP32 start of 1/R only.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "g64tables.h"

#if defined(__CUDACC__)
#define G64_HD __host__ __device__ __forceinline__
#define G64_SLOW __host__ __device__ __noinline__
#else
#define G64_HD inline
#define G64_SLOW inline
#endif

namespace g64 {

constexpr int QUARTER = 1024;            // table steps per quarter turn
constexpr int TABLE = QUARTER + 1;       // entries
constexpr double STEPS_PER_RADIAN = 651.89864690440329530934789477382;  // 4096 / (2 pi)

// sin of a table point and the same as a float pair
struct Entry {
  double v;
  float hi, lo;
};

#if defined(__CUDACC__)
static __device__ const double sin_table_dev[TABLE] = G64_SIN_TABLE_INIT;
#endif
static const double sin_table_host[TABLE] = G64_SIN_TABLE_INIT;

// the wavenumber as the evaluation takes it: |k| in steps per unit length, split
struct Wave {
  double k;      // |k|
  double steps;  // |k| 4096 / (2 pi), rounded
  float rest;    // what the rounding left
};
inline Wave make_wave(double gi) {
  Wave w;
  w.k = fabs(gi);
  const long double s = (long double)w.k * 651.89864690440329530934789477382L;
  w.steps = (double)s;
  w.rest = (float)(s - (long double)w.steps);
  return w;
}

G64_HD uint64_t bits(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
G64_HD double from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
G64_HD uint32_t fbits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}
G64_HD float from_fbits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}
#if defined(__CUDA_ARCH__)
G64_HD float fadd(float a, float b) { return __fadd_rn(a, b); }
G64_HD float fsub(float a, float b) { return __fsub_rn(a, b); }
G64_HD float fmul(float a, float b) { return __fmul_rn(a, b); }
#else
G64_HD float fadd(float a, float b) { return a + b; }
G64_HD float fsub(float a, float b) { return a - b; }
G64_HD float fmul(float a, float b) { return a * b; }
#endif

// h + l as a double, built from the bits: h exactly, l added to the mantissa as an integer number
// of its units (|l| at most a few ulp of h); h = 0: 0
G64_HD double pair_to_double(float h, float l) {
  const uint32_t u = fbits(h), e = (u >> 23) & 0xFF;
  const uint64_t m = ((uint64_t)(e + 896) << 52) | ((uint64_t)(u & 0x7FFFFFu) << 29);
  // l in units of the double's last place, 2^(e - 127 - 52)
  const float unit = e >= 52 ? from_fbits((306u - e) << 23) : 0.f;
#if defined(__CUDA_ARCH__)
  int d = __float2int_rn(fmul(l, unit));
#else
  int d = (int)lrintf(l * unit);
#endif
  d = (int32_t)u < 0 ? -d : d;
  // below a power of two the last place is half as large
  if ((u & 0x7FFFFFu) == 0 && d < 0) d *= 2;
  const uint64_t r = m + (uint64_t)(int64_t)d;
  return e == 0 ? 0.0 : from_bits(r | ((uint64_t)(u >> 31) << 63));
}
G64_HD double half(double x) { return from_bits(bits(x) - (1ull << 52)); }  // x / 2, normal range

// (ah + al) (x + y) left unnormalised
G64_HD void pair_mul(float ah, float al, float x, float y, float& h, float& l) {
  h = fmul(ah, x);
  l = fadd(fmaf(ah, x, -h), fmaf(ah, y, fmul(al, x)));
}

struct Value {
  double iR, R, c, s;  // 1/R, R, cos(|k| R), sin(|k| R)
};

G64_SLOW Value eval_slow(double R2, double k) {
  Value v;
#if defined(__CUDA_ARCH__)
  v.iR = rsqrt(R2);
#else
  v.iR = 1.0 / sqrt(R2);
#endif
  v.R = R2 * v.iR;
#if defined(__CUDA_ARCH__)
  sincos(k * v.R, &v.s, &v.c);
#else
  v.s = sin(k * v.R);
  v.c = cos(k * v.R);
#endif
  return v;
}

// 1/sqrt(R2) and sqrt(R2) for R2 in [2^-100, 2^90]
G64_HD void inv_sqrt(double R2, double& iR, double& R) {
  const uint64_t u = bits(R2);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const uint32_t f = ((hi - (896u << 20)) << 3) | (lo >> 29);
  const float a = from_fbits(f);  // R2 truncated, and the rest
  const float al = fmul(fmul((float)(int)(lo & 0x1FFFFFFFu), 1.862645149230957e-09f), from_fbits((f & 0x7F800000u) - (23u << 23)));
#if defined(__CUDA_ARCH__)
  const float y0 = rsqrtf(a);
#else
  const float y0 = 1.f / sqrtf(a);
#endif
  const float p = fmul(y0, y0), pl = fmaf(y0, y0, -p);
  const float q = fmul(a, p);
  const float e = fsub(fsub(1.f, q), fadd(fmaf(a, p, -q), fmaf(a, pl, fmul(al, p))));  // 1 - R2 y0^2
  const double y = pair_to_double(y0, fmul(fmul(y0, e), fmaf(0.375f, e, 0.5f)));
  const double g = R2 * y;
  const double r = fma(-g, y, 1.0);
  iR = fma(r, half(y), y);
  R = fma(r, half(g), g);
}

// what the fraction of a step, f in [-1/2, 1/2) as the 64-bit fixed-point number fh:fl (plus rest), adds
// to the table point's sine and cosine A, B: float pairs (sh, sl), (ch, cl) with |sh| at least |sl|
G64_HD void correction(uint32_t fh, uint32_t fl, float rest, float Ah, float Al, float Bh, float Bl, float& sh, float& sl,
                       float& ch, float& cl) {
  // the fraction as 24 + 32 bits
  const float fa = fmul((float)(int32_t)(fh & 0xFFFFFF00u), 2.3283064365386963e-10f);
  const float fb = fmaf((float)((fh << 24) | (fl >> 8)), 1.3877787807814457e-17f, rest);
  const float th = fmul(fa, G64_STEP_HI);
  const float tl = fadd(fmaf(fa, G64_STEP_HI, -th), fmaf(fa, G64_STEP_LO, fmul(fb, G64_STEP_HI)));
  const float p = fmul(th, th);
  const float pl = fmaf(th, th, -p) + 2.f * fmul(th, tl);
  // cos t - 1 and sin t
  const float kh = fmul(-0.5f, p), kl = fmaf(-0.5f, pl, fmul(fmul(p, p), 1.f / 24.f));
  const float ul = fmaf(fmul(th, p), fmaf(p, 1.f / 120.f, -1.f / 6.f), tl);
  float h1, l1, h2, l2;
  pair_mul(Bh, Bl, th, ul, h1, l1);
  pair_mul(Ah, Al, kh, kl, h2, l2);
  float h = fadd(h1, h2);
  float bb = fsub(h, h1);
  float l = fadd(fadd(fsub(h1, fsub(h, bb)), fsub(h2, bb)), fadd(l1, l2));
  sh = fadd(h, l);
  sl = fsub(l, fsub(sh, h));
  pair_mul(Bh, Bl, kh, kl, h1, l1);
  pair_mul(-Ah, -Al, th, ul, h2, l2);
  h = fadd(h1, h2);
  bb = fsub(h, h1);
  l = fadd(fadd(fsub(h1, fsub(h, bb)), fsub(h2, bb)), fadd(l1, l2));
  ch = fadd(h, l);
  cl = fsub(l, fsub(ch, h));
}

// cos and sin of n + f steps
G64_HD void rotate(uint32_t n, uint32_t fh, uint32_t fl, float rest, const Entry* tab, double& c, double& s) {
  const int i = (int)(n & (QUARTER - 1)), q = (int)(n >> 10) & 3;
  const Entry A = tab[i], B = tab[QUARTER - i];
  float sh, sl, ch, cl;
  correction(fh, fl, rest, A.hi, A.lo, B.hi, B.lo, sh, sl, ch, cl);
  const double s0 = A.v + pair_to_double(sh, sl), c0 = B.v + pair_to_double(ch, cl);
  // quarter turns
  const uint64_t us = bits((q & 1) ? c0 : s0), uc = bits((q & 1) ? s0 : c0);
  s = from_bits(us ^ ((uint64_t)(q >> 1) << 63));
  c = from_bits(uc ^ ((uint64_t)(((q + 1) >> 1) & 1) << 63));
}

// cos and sin of phi steps (+ rest steps) for phi in [64, 2^30)
G64_HD void turn(double phi, float rest, const Entry* tab, double& c, double& s) {
  const uint64_t u = bits(phi);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const int e = (int)(hi >> 20) - 1023;  // 6 .. 29
  // the mantissa at the top of 64 bits: integer part above bit 63 - e, fraction below
  const uint32_t xh = ((hi << 11) | (lo >> 21)) | 0x80000000u, xl = lo << 11;
  const uint32_t fh = (xh << (e + 1)) | (xl >> (31 - e)), fl = xl << (e + 1);
  rotate((xh >> (31 - e)) + (fh >> 31), fh, fl, rest, tab, c, s);
}

// the same for any phi (+ rest) with |phi| < 2^30, to 2^-52 absolutely (a small sine keeps no
// relative accuracy); false: out of range
G64_HD bool turn_signed(double phi, float rest, const Entry* tab, double& c, double& s) {
  const uint64_t u = bits(phi);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const int e = (int)((hi >> 20) & 0x7FF) - 1023;
  if (e > 29) return false;
  const uint64_t x = ((uint64_t)(((hi << 11) | (lo >> 21)) | 0x80000000u) << 32) | (lo << 11);
  const uint64_t f = e >= 0 ? x << (e + 1) : (e > -64 ? x >> (-1 - e) : 0);
  const uint32_t n0 = e >= 0 ? (uint32_t)(x >> 32) >> (31 - e) : 0u;
  rotate(n0 + (uint32_t)(f >> 63), (uint32_t)(f >> 32), (uint32_t)f, (u >> 63) ? -rest : rest, tab, c, s);
  s = from_bits(bits(s) ^ (u & 0x8000000000000000ull));
  return true;
}

G64_HD Value eval(double R2, const Wave& w, const Entry* tab) {
  Value v;
  if ((uint32_t)((uint32_t)(bits(R2) >> 52) - 923u) > 190u) return eval_slow(R2, w.k);
  inv_sqrt(R2, v.iR, v.R);
  if (w.k == 0.0) {  // static kernels
    v.c = 1.0;
    v.s = 0.0;
    return v;
  }
  const double phi = v.R * w.steps;
  if ((uint32_t)((uint32_t)(bits(phi) >> 52) - 1029u) > 23u) return eval_slow(R2, w.k);
  const float rest = fmul(w.rest, from_fbits((uint32_t)(((bits(v.R) >> 32) - (896ull << 20)) << 3)));
  turn(phi, rest, tab, v.c, v.s);
  return v;
}

// ---- the same in 64-bit fixed point ---------------------------------------------------------
// Sums of kernel values times rule weights need no exponent of their own: as integers they cost two
// instructions per addition and about a dozen per product where the FP64 pipe takes 64 issue slots
// for either.  Values are int64 with 62 fractional bits.

// round(x 2^62) of a float pair, |h| < 2^-9
G64_HD int64_t pair_to_fixed(float h, float l) {
#if defined(__CUDA_ARCH__)
  const int i = __float2int_rn(fmul(h, 274877906944.f));  // 2^38
#else
  const int i = (int)lrintf(h * 274877906944.f);
#endif
  const float r = fmaf(-(float)i, 3.637978807091713e-12f, h) + l;
#if defined(__CUDA_ARCH__)
  const int k = __float2int_rn(fmul(r, 4611686018427387904.f));
#else
  const int k = (int)lrintf(r * 4611686018427387904.f);
#endif
  return ((int64_t)i << 24) + k;
}
// x 2^(62 - e) of a double with |x| < 2^e, truncated
G64_HD int64_t to_fixed(double x, int e) {
  const uint64_t u = bits(x);
  const int E = (int)((u >> 52) & 0x7FF) - 1023;
  const uint64_t m = E == -1023 ? 0 : (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = 10 + E - e;  // < 10
  const uint64_t v = sh >= 0 ? m << (sh & 63) : (sh > -64 ? m >> (-sh & 63) : 0);
  return (u >> 63) ? -(int64_t)v : (int64_t)v;
}
// x 2^e of an integer as a double, rounded to nearest (ties up); no FP64 instruction
G64_HD double from_fixed(int64_t x, int e) {
  const uint64_t sgn = (uint64_t)x & 0x8000000000000000ull;
  const uint64_t u = x < 0 ? 0ull - (uint64_t)x : (uint64_t)x;
  if (u == 0) return 0.0;
#if defined(__CUDA_ARCH__)
  const int lz = __clzll((long long)u);
#else
  const int lz = __builtin_clzll(u);
#endif
  const uint64_t m = u << lz;
  const uint64_t r = (m >> 11) + ((m >> 10) & 1);  // 2^52 .. 2^53
  return from_bits(sgn | (((uint64_t)(1023 + 63 - lz + e - 1) << 52) + r));
}
G64_HD int64_t mulhi(int64_t a, int64_t b) {
#if defined(__CUDA_ARCH__)
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}

struct EntryX {
  int64_t v;  // sin 2^62
  float hi, lo;
};
G64_HD EntryX to_entryx(double x) {
  const float h = (float)x;
  return EntryX{x >= 1.0 ? (int64_t)1 << 62 : to_fixed(x, 0), h, (float)(x - (double)h)};
}
struct ValueX {
  double iR;     // 1/R
  int64_t c, s;  // cos(|k| R), sin(|k| R)
};
// false: R2 or the angle out of range (below 4 steps, kR = 0.0061, the integer sine would lose relative accuracy)
G64_HD bool eval_fixed(double R2, const Wave& w, const EntryX* tab, ValueX& v) {
  if ((uint32_t)((uint32_t)(bits(R2) >> 52) - 923u) > 190u) return false;
  double R;
  inv_sqrt(R2, v.iR, R);
  const double phi = R * w.steps;
  const uint64_t u = bits(phi);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const int e = (int)(hi >> 20) - 1023;
  if ((uint32_t)(e - 2) > 27u) return false;  // 4 <= phi < 2^30
  const float rest = fmul(w.rest, from_fbits((uint32_t)(((bits(R) >> 32) - (896ull << 20)) << 3)));
  const uint32_t xh = ((hi << 11) | (lo >> 21)) | 0x80000000u, xl = lo << 11;
  const uint32_t fh = (xh << (e + 1)) | (xl >> (31 - e)), fl = xl << (e + 1);
  const uint32_t n = (xh >> (31 - e)) + (fh >> 31);
  const int i = (int)(n & (QUARTER - 1)), q = (int)(n >> 10) & 3;
  const EntryX A = tab[i], B = tab[QUARTER - i];
  float sh, sl, ch, cl;
  correction(fh, fl, rest, A.hi, A.lo, B.hi, B.lo, sh, sl, ch, cl);
  const int64_t s0 = A.v + pair_to_fixed(sh, sl), c0 = B.v + pair_to_fixed(ch, cl);
  const int64_t us = (q & 1) ? c0 : s0, uc = (q & 1) ? s0 : c0;
  v.s = (q >> 1) ? -us : us;
  v.c = (((q + 1) >> 1) & 1) ? -uc : uc;
  return true;
}

#if defined(__CUDACC__)
// the table into shared memory, by the whole CTA (the caller synchronises)
__device__ __forceinline__ void load_table(Entry* tab) {
  for (int i = threadIdx.x; i < TABLE; i += blockDim.x) {
    const double x = sin_table_dev[i];
    const float h = (float)x;
    tab[i] = Entry{x, h, (float)(x - (double)h)};
  }
}
__device__ __forceinline__ void load_table(EntryX* tab) {
  for (int i = threadIdx.x; i < TABLE; i += blockDim.x) tab[i] = to_entryx(sin_table_dev[i]);
}
#endif

}  // namespace g64
