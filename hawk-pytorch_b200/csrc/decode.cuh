// What the single-token kernels share: loads of a predecessor's results, asynchronous copies to shared memory, and the
// launch of the recurrent branch's step.
#pragma once

#include "common.cuh"

namespace hawk {

// 8 consecutive elements written by the preceding kernel (16-byte aligned), as fp32
__device__ __forceinline__ void load_dep8(const float* p, float (&v)[8]) {
  const uint4 a = ld_dep16(p), b = ld_dep16(p + 4);
  v[0] = __uint_as_float(a.x); v[1] = __uint_as_float(a.y); v[2] = __uint_as_float(a.z); v[3] = __uint_as_float(a.w);
  v[4] = __uint_as_float(b.x); v[5] = __uint_as_float(b.y); v[6] = __uint_as_float(b.z); v[7] = __uint_as_float(b.w);
}
__device__ __forceinline__ void load_dep8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 a = ld_dep16(p);
  const float2 q0 = unpack_bf16x2(a.x), q1 = unpack_bf16x2(a.y), q2 = unpack_bf16x2(a.z), q3 = unpack_bf16x2(a.w);
  v[0] = q0.x; v[1] = q0.y; v[2] = q1.x; v[3] = q1.y; v[4] = q2.x; v[5] = q2.y; v[6] = q3.x; v[7] = q3.y;
}
// one element of the same
__device__ __forceinline__ float load_dep(const float* p) { return *static_cast<const volatile float*>(p); }
__device__ __forceinline__ float load_dep(const __nv_bfloat16* p) {
  const unsigned short u = *reinterpret_cast<const volatile unsigned short*>(p);
  return __uint_as_float((uint32_t)u << 16);
}

// v rounded to T's precision
template <typename T>
__device__ __forceinline__ float from_float_round(float v) { return to_float(from_float<T>(v)); }

__device__ __forceinline__ void copy_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// hawk_decode_block_step without the argument checks; pdl: as a programmatic dependent launch (the gate weights, biases, taps
// and Lambda are then not written by the kernel before it)
int block_step(const void* xy, int64_t ld_xy, void* conv_state, const float* cw, const float* cb, const void* wx, const void* wa,
               const float* bx, const float* ba, const float* lam, void* state, void* out, int B, int R, int bw, int W, int dtype,
               int state_dtype, int weight_dtype, bool pdl, cudaStream_t st);

}  // namespace hawk
