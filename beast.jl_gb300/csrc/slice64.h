// slice64.h -- the digits of the sliced FP64 update (tc_gemm64.cu), host and device.
//
// A row (or column) of FP64 values is scaled by a power of two 2^-e with |x| < 2^e for its largest
// magnitude, taken to the fixed-point integer X = round(x 2^(55 - e)), |X| <= 2^55, and written
// with SLICES balanced digits of 7 bits,
//   x 2^-e = sum_i d_i 2^(-6 - 7 i) + r,   -64 <= d_i <= 64,   |r| <= 2^-56,
// each exactly an FP16 number.  A product of two digits is at most 2^12, so a sum of up to 4096 of
// them is an integer of at most 2^24 that FP32 accumulation holds exactly, whatever the order.
//
// Balance.  The digits cut a value relative to its row's largest, so a sum over k of a_ik b_kj whose
// terms meet large a with small b (rows of a matrix in different units: a_ik ~ d_i / d_k, b_kj ~ d_k)
// would lose what FP64 keeps.  The sum is therefore taken over (a_ik 2^-s_k) (b_kj 2^s_k) with 2^s_k
// the power of two above the largest |a_ik| of column k: exact, and the same for every scaling of the
// rows and columns by powers of two.
// Spread.  What no such scaling levels (blocks of unknowns that are hardly coupled) is measured: the
// sum S_ij over k of p_ik q_kj, p and q the magnitudes relative to 2^e of their row and column.  The
// digits' error is at most about 2^-54 of the row's times the column's largest value, so relative to
// sum |a_ik b_kj| it stays near FP64's own where S_ij is not far below one (and relative to the entry the sum is
// subtracted from where that is not).
#pragma once
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define SL_HD __host__ __device__ __forceinline__
#else
#define SL_HD inline
#endif

namespace slice64 {

constexpr int SLICES = 8;
constexpr int EXP_NONFINITE = 1 << 20;  // row exponent of a row that holds an infinity or a NaN

SL_HD uint64_t bits_of(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}

// the top word of |x|: ordered like |x| up to its low 32 bits, 0x7FF00000 and above: not finite
SL_HD uint32_t abs_hi(double x) { return (uint32_t)(bits_of(x) >> 32) & 0x7FFFFFFFu; }

// the exponent e of a row whose largest abs_hi is hi: every |x| of the row < 2^e (subnormal rows
// take the smallest normal exponent; an all-zero row is one of them)
SL_HD int row_exponent(uint32_t hi) {
  const int E = (int)(hi >> 20);
  if (E >= 2047) return EXP_NONFINITE;
  return (E > 0 ? E : 1) - 1022;
}

// s_k of a column whose largest abs_hi is hi (0 for a column that holds an infinity or a NaN)
SL_HD int balance_exponent(uint32_t hi) {
  const int e = row_exponent(hi);
  return e == EXP_NONFINITE ? 0 : e;
}
// the exponent of x 2^s as a key that is ordered like it (a zero below every other value, what is not
// finite above), and the exponent e of a row from its largest key: every |x| 2^s of the row < 2^e
constexpr int KEY_ZERO = -(1 << 20);
SL_HD int scaled_key(double x, int s) {
  const int E = (int)(abs_hi(x) >> 20);
  if (E >= 2047) return EXP_NONFINITE;
  return (bits_of(x) << 1) == 0 ? KEY_ZERO : (E > 0 ? E : 1) - 1022 + s;
}
SL_HD int key_exponent(int key) {
  return key >= EXP_NONFINITE / 2 ? EXP_NONFINITE : (key == KEY_ZERO ? -1021 : key);
}

// round(x 2^(b - e)), ties up in magnitude; |x| < 2^e, b <= 62
SL_HD int64_t fixed_point(double x, int e, int b) {
  const uint64_t u = bits_of(x);
  const int E = (int)((u >> 52) & 0x7FF);
  const uint64_t m = (u & 0xFFFFFFFFFFFFFull) | (E ? 1ull << 52 : 0ull);
  const int sh = (E ? E : 1) - 1075 + b - e;  // x = m 2^(E - 1075); sh <= b - 53
  uint64_t X;
  if (sh >= 0)
    X = m << sh;
  else if (sh > -56)
    X = (m + (1ull << (-sh - 1))) >> -sh;
  else
    X = 0;
  return (u >> 63) ? -(int64_t)X : (int64_t)X;
}

// the fixed-point number of the eight digits, and of nine
SL_HD int64_t fixed55(double x, int e) { return fixed_point(x, e, 55); }
SL_HD int64_t fixed62(double x, int e) { return fixed_point(x, e, 62); }

// the digits of X, most significant first
SL_HD void digits(int64_t X, int d[SLICES]) {
#pragma unroll
  for (int i = SLICES - 1; i > 0; --i) {
    d[i] = (int)((X + 64) & 127) - 64;
    X = (X - d[i]) >> 7;
  }
  d[0] = (int)X;
}

// the nine digits of X = fixed62: the ninth is taken off, the rest is the eight digits' number
SL_HD void digits9(int64_t X, int d[SLICES + 1]) {
  d[SLICES] = (int)((X + 64) & 127) - 64;
  digits((X - d[SLICES]) >> 7, d);
}

// the magnitude of a complex value from its two parts (fixed62), relative to 2^e: 2^-24 at least (the smallest FP16
// number) unless both are exactly zero, at most 1
constexpr float SPREAD_MIN = 0x1p-24f;
SL_HD float spread_magnitude(int64_t X, int64_t Y, bool zero) {
  const int64_t x = X < 0 ? -X : X, y = Y < 0 ? -Y : Y;
  const float p = (float)(int32_t)((x > y ? x : y) >> 32) * 0x1p-30f;
  return zero ? 0.f : (p > SPREAD_MIN ? p : SPREAD_MIN);
}
// An entry with a sum 0 < S < 2^-SPREAD_BITS that is itself below the same part of its scale needs the ninth digit,
// below 2^-SPREAD_BITS_FP64 the FP64 units.  (An FP64 update rounds to 2^-53 of the entry or the sum, whichever is
// larger; eight digits cut at 2^-55 of the scale, nine at 2^-62.)  Two blocks of unknowns coupled by 2^-9 lose a factor
// of 6 in the accuracy of the weak one at these limits; at 2^-13 it would be a hundred.
constexpr int SPREAD_BITS = 10, SPREAD_BITS_FP64 = 17;
// max(|x|, |y|) < 2^(e - bits)
SL_HD bool spread_small(double x, double y, int e, int bits) {
  const uint32_t a = abs_hi(x), b = abs_hi(y);
  return (int)((a > b ? a : b) >> 20) - 1022 <= e - bits;
}

// the FP64 value -D 2^sh of an integer-valued FP32 number D, built from its bits (a conversion
// would run on the FP64 pipe); sh >= EXP_NONFINITE / 2: NaN; results below the normal range: 0
SL_HD double neg_scaled(float D, int sh) {
  uint32_t f;
#if defined(__CUDA_ARCH__)
  f = __float_as_uint(D);
#else
  memcpy(&f, &D, 4);
#endif
  const int E = (int)((f >> 23) & 0xFF) + 896 + sh;
  uint32_t hi = (~f & 0x80000000u) | ((uint32_t)E << 20) | ((f >> 3) & 0xFFFFFu), lo = f << 29;
  if (E >= 2047) {
    hi = (~f & 0x80000000u) | 0x7FF00000u;
    lo = 0;
  }
  if ((f << 1) == 0 || E <= 0) hi = lo = 0;
  if (sh >= EXP_NONFINITE / 2) hi = 0x7FF80000u;
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double r;
  memcpy(&r, &u, 8);
  return r;
#endif
}

}  // namespace slice64
