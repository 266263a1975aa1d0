// Two floats in one 64-bit register pair, and the packed FMA on them: what the 32-bit kernels (gemm_f32.cu, gemm_f32x3.cu,
// attention_f32.cu) share.
#pragma once

typedef unsigned long long f32x2;                // the lower one in the low word

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 pair2(float lo, float hi) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 split2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  const float2 r = split2(v);
  return r.x + r.y;
}
// Two such pairs out of shared memory.
__device__ __forceinline__ ulonglong2 lds_pair(unsigned addr) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];\n" : "=l"(v.x), "=l"(v.y) : "r"(addr));
  return v;
}
