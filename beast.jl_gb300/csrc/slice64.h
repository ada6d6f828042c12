// slice64.h -- the digits of the sliced FP64 update (tc_gemm64.cu), host and device.
//
// A row (or column) of FP64 values is scaled by a power of two 2^-e with |x| < 2^e for its largest
// magnitude, taken to the fixed-point integer X = round(x 2^(55 - e)), |X| <= 2^55, and written
// with SLICES balanced digits of 7 bits,
//   x 2^-e = sum_i d_i 2^(-6 - 7 i) + r,   -64 <= d_i <= 64,   |r| <= 2^-56,
// each exactly an FP16 number.  A product of two digits is at most 2^12, so a sum of up to 4096 of
// them is an integer of at most 2^24 that FP32 accumulation holds exactly, whatever the order.
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

// round(x 2^(55 - e)), ties up in magnitude; |x| < 2^e
SL_HD int64_t fixed55(double x, int e) {
  const uint64_t u = bits_of(x);
  const int E = (int)((u >> 52) & 0x7FF);
  const uint64_t m = (u & 0xFFFFFFFFFFFFFull) | (E ? 1ull << 52 : 0ull);
  const int sh = (E ? E : 1) - 1020 - e;  // x = m 2^(E - 1075); sh <= 2
  uint64_t X;
  if (sh >= 0)
    X = m << sh;
  else if (sh > -56)
    X = (m + (1ull << (-sh - 1))) >> -sh;
  else
    X = 0;
  return (u >> 63) ? -(int64_t)X : (int64_t)X;
}

// the digits of X, most significant first
SL_HD void digits(int64_t X, int d[SLICES]) {
#pragma unroll
  for (int i = SLICES - 1; i > 0; --i) {
    d[i] = (int)((X + 64) & 127) - 64;
    X = (X - d[i]) >> 7;
  }
  d[0] = (int)X;
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
