// Device code that the two strict-FP32 kernels share (conv_fp32.cu, conv_fp32_wide.cu).
#pragma once

#include "ptx.cuh"

namespace gieb {

// 16-byte asynchronous copy global -> shared (both addresses 16-byte aligned); `bytes` of the source are read, the rest is zero-filled.
__device__ __forceinline__ void cp_async16(void* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// Two FP32 values in one 64-bit register: the operands of fma.rn.f32x2.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }

}  // namespace gieb
