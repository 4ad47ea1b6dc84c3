// AdamW update of fp32 parameter tensors in a single pass, optionally emitting the bf16 copy of the
// updated weights that the next step's bf16 GEMMs consume.  Training with torch.optim.AdamW under bf16
// autocast makes an optimiser pass over p, g, m, v and then, at the next forward, a separate
// fp32 -> bf16 cast pass per weight.  Here the cast rides on the update: 28 bytes per element read or
// written for the update, 2 more for the bf16 copy, and nothing is touched again.
#include "common.cuh"

namespace hawk {

struct AdamwArgs {
  float lr, beta1, beta2, eps, decay_factor;  // decay_factor = 1 - lr * weight_decay
  float step_size;                            // lr / (1 - beta1^t)
  float inv_sqrt_bc2;                         // 1 / sqrt(1 - beta2^t)
};

__device__ __forceinline__ float adamw_one(float p, float g, float& m, float& v, const AdamwArgs& a) {
  p *= a.decay_factor;
  m = fmaf(a.beta1, m, (1.f - a.beta1) * g);
  v = fmaf(a.beta2, v, (1.f - a.beta2) * g * g);
  const float denom = fmaf(sqrtf(v), a.inv_sqrt_bc2, a.eps);
  return p - a.step_size * (m / denom);
}

// One launch updates up to kAdamwTensors tensors: a model of 42 M parameters in 55 tensors spent 328 us in as many launches,
// most of them a wave of a few blocks that start, read once and drain.  A block takes kAdamwChunk consecutive elements of
// one tensor; the table with the tensors' addresses and first blocks comes as a kernel parameter (under 4 KB).
constexpr int kAdamwTensors = 64, kAdamwChunk = 8192;

struct AdamwTable {
  hawk_adamw_tensor t[kAdamwTensors];
  uint32_t first[kAdamwTensors + 1];  // first block of each tensor
  uint8_t vec[kAdamwTensors];         // 16-byte accesses
  int count;
};

__global__ void __launch_bounds__(256) adamw_kernel(const __grid_constant__ AdamwTable tab, AdamwArgs a) {
  int lo = 0, hi = tab.count;  // the tensor whose blocks hold this one
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x >= tab.first[mid]) lo = mid; else hi = mid;
  }
  const hawk_adamw_tensor& t = tab.t[lo];
  const int64_t i0 = (int64_t)(blockIdx.x - tab.first[lo]) * kAdamwChunk;
  const int64_t n = t.n - i0 < kAdamwChunk ? t.n - i0 : kAdamwChunk;
  float* p = t.p + i0;
  const float* g = t.g + i0;
  float* m = t.m + i0;
  float* v = t.v + i0;
  __nv_bfloat16* p16 = t.p_bf16 ? static_cast<__nv_bfloat16*>(t.p_bf16) + i0 : nullptr;
  int64_t done = 0;
  if (tab.vec[lo]) {
    const int nvec = (int)(n / 4);
#pragma unroll 2
    for (int i = threadIdx.x; i < nvec; i += 256) {
      float4 pv = reinterpret_cast<float4*>(p)[i];
      const float4 gv = __ldg(reinterpret_cast<const float4*>(g) + i);
      float4 mv = reinterpret_cast<float4*>(m)[i], vv = reinterpret_cast<float4*>(v)[i];
      pv.x = adamw_one(pv.x, gv.x, mv.x, vv.x, a);
      pv.y = adamw_one(pv.y, gv.y, mv.y, vv.y, a);
      pv.z = adamw_one(pv.z, gv.z, mv.z, vv.z, a);
      pv.w = adamw_one(pv.w, gv.w, mv.w, vv.w, a);
      reinterpret_cast<float4*>(p)[i] = pv;
      reinterpret_cast<float4*>(m)[i] = mv;
      reinterpret_cast<float4*>(v)[i] = vv;
      if (p16 != nullptr)
        reinterpret_cast<uint2*>(p16)[i] = make_uint2(pack_bf16x2(pv.x, pv.y), pack_bf16x2(pv.z, pv.w));
    }
    done = (int64_t)nvec * 4;
  }
  for (int64_t i = done + threadIdx.x; i < n; i += 256) {  // ragged tail, or a tensor at an odd address
    float mm = m[i], vv = v[i];
    const float pn = adamw_one(p[i], g[i], mm, vv, a);
    p[i] = pn; m[i] = mm; v[i] = vv;
    if (p16 != nullptr) p16[i] = __float2bfloat16(pn);
  }
}

}  // namespace hawk

using namespace hawk;

extern "C" int hawk_adamw_multi(const hawk_adamw_tensor* tensors, int count, float lr, float beta1, float beta2, float eps,
                                float weight_decay, int64_t step, void* stream) {
  HAWK_REQUIRE(tensors, HAWK_ERR_NULL);
  HAWK_REQUIRE(count >= 1 && step >= 1, HAWK_ERR_SHAPE);
  for (int i = 0; i < count; ++i) {
    const hawk_adamw_tensor& t = tensors[i];
    HAWK_REQUIRE(t.p && t.g && t.m && t.v, HAWK_ERR_NULL);
    HAWK_REQUIRE(t.n >= 1 && t.n <= (1LL << 40), HAWK_ERR_SHAPE);
    HAWK_REQUIRE(aligned(t.p, 4) && aligned(t.g, 4) && aligned(t.m, 4) && aligned(t.v, 4) && aligned(t.p_bf16, 2), HAWK_ERR_ALIGN);
  }
  AdamwArgs a;
  a.lr = lr;
  a.beta1 = beta1;
  a.beta2 = beta2;
  a.eps = eps;
  a.decay_factor = 1.f - lr * weight_decay;
  const double bc1 = 1.0 - pow((double)beta1, (double)step), bc2 = 1.0 - pow((double)beta2, (double)step);
  a.step_size = (float)((double)lr / bc1);
  a.inv_sqrt_bc2 = (float)(1.0 / sqrt(bc2));
  for (int i0 = 0; i0 < count;) {
    AdamwTable tab;
    uint32_t blocks = 0;
    int k = 0;
    for (; k < kAdamwTensors && i0 + k < count; ++k) {
      const hawk_adamw_tensor& t = tensors[i0 + k];
      const int64_t need = (t.n + kAdamwChunk - 1) / kAdamwChunk;
      if (need > (int64_t)0x7fffffff - blocks) break;  // the next launch's
      tab.t[k] = t;
      tab.first[k] = blocks;
      tab.vec[k] = aligned(t.p, 16) && aligned(t.g, 16) && aligned(t.m, 16) && aligned(t.v, 16) && aligned(t.p_bf16, 8);
      blocks += (uint32_t)need;
    }
    tab.first[k] = blocks;
    tab.count = k;
    adamw_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(tab, a);
    const int rc = launch_status();
    if (rc != HAWK_OK) return rc;
    i0 += k;
  }
  return HAWK_OK;
}

extern "C" int hawk_adamw_step(float* p, const float* g, float* m, float* v, void* p_bf16, int64_t n, float lr,
                               float beta1, float beta2, float eps, float weight_decay, int64_t step, void* stream) {
  const hawk_adamw_tensor one = {p, g, m, v, p_bf16, n};
  return hawk_adamw_multi(&one, 1, lr, beta1, beta2, eps, weight_decay, step, stream);
}
