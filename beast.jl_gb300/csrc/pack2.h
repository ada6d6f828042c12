// Two FP32 values in one 64-bit register pair and the arithmetic on both at once (sm_100 and later).
// A packed instruction does two lanes' work in one issue slot; the FP32 pipes do not get faster by it
// (measured on GB300: 238 fused multiply-adds per ns and SM packed, 215 single; with half as many
// integer instructions between them 200 against 155).  Kernels whose issue slots are full of FP32
// instructions gain.  Each lane is rounded as the single instruction rounds it.
#pragma once

namespace pk {

struct f2 {
  float2 v;
};
__device__ __forceinline__ f2 make(float a, float b) { return f2{make_float2(a, b)}; }
__device__ __forceinline__ f2 both(float a) { return make(a, a); }
__device__ __forceinline__ float lo(f2 a) { return a.v.x; }
__device__ __forceinline__ float hi(f2 a) { return a.v.y; }
__device__ __forceinline__ f2 add(f2 a, f2 b) { return f2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ f2 sub(f2 a, f2 b) { return f2{__fadd2_rn(a.v, make_float2(-b.v.x, -b.v.y))}; }
__device__ __forceinline__ f2 mul(f2 a, f2 b) { return f2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) { return f2{__ffma2_rn(a.v, b.v, c.v)}; }

}  // namespace pk
