// What the single-token kernels share: loads of a predecessor's results, asynchronous copies to shared memory, and the
// launch of the recurrent branch's step.
#pragma once

#include "common.cuh"

namespace hawk {

// 8 elements from their 16-byte words (one of bf16, two of fp32)
__device__ __forceinline__ void unpack8(const uint4 (&r)[1], float (&v)[8]) {
  const float2 q0 = unpack_bf16x2(r[0].x), q1 = unpack_bf16x2(r[0].y), q2 = unpack_bf16x2(r[0].z), q3 = unpack_bf16x2(r[0].w);
  v[0] = q0.x; v[1] = q0.y; v[2] = q1.x; v[3] = q1.y; v[4] = q2.x; v[5] = q2.y; v[6] = q3.x; v[7] = q3.y;
}
__device__ __forceinline__ void unpack8(const uint4 (&r)[2], float (&v)[8]) {
  v[0] = __uint_as_float(r[0].x); v[1] = __uint_as_float(r[0].y); v[2] = __uint_as_float(r[0].z); v[3] = __uint_as_float(r[0].w);
  v[4] = __uint_as_float(r[1].x); v[5] = __uint_as_float(r[1].y); v[6] = __uint_as_float(r[1].z); v[7] = __uint_as_float(r[1].w);
}
// and back, rounding to the type
__device__ __forceinline__ void pack8(const float (&v)[8], uint4 (&r)[1]) {
  r[0] = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ void pack8(const float (&v)[8], uint4 (&r)[2]) {
  r[0] = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  r[1] = make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
}
// 8 consecutive elements written by the preceding kernel (16-byte aligned), as fp32
__device__ __forceinline__ void load_dep8(const float* p, float (&v)[8]) {
  const uint4 r[2] = {ld_dep16(p), ld_dep16(p + 4)};
  unpack8(r, v);
}
__device__ __forceinline__ void load_dep8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 r[1] = {ld_dep16(p)};
  unpack8(r, v);
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
