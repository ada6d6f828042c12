// Two FP32 values in one 64-bit register pair and the arithmetic on both at once (sm_100 and later).
// A packed instruction does two lanes' work in one issue slot; the FP32 pipes do not get faster by it
// (measured on GB300: 238 fused multiply-adds per ns and SM packed, 215 single; with half as many
// integer instructions between them 200 against 155).  Kernels whose issue slots are full of FP32
// instructions gain.  Each lane is rounded as the single instruction rounds it.
#pragma once

namespace pk {

struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 make(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 both(float a) { return make(a, a); }
__device__ __forceinline__ void split(f2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ float lo(f2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(f2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ f2 add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

}  // namespace pk
