// Packed fp32 arithmetic and the bf16 conversions around it, for the element-wise parts of the tensor-core kernels.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace tc {

// Two fp32 values per register pair: the Blackwell f32x2 instructions do two IEEE operations per issue slot.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void split2(f32x2 v, float* a, float* b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t bf16_pair(f32x2 v) {
  float a, b;
  split2(v, &a, &b);
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ f32x2 from_bf16_pair(uint32_t v) { return pair2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }

// The largest of three in one instruction.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

}  // namespace tc
