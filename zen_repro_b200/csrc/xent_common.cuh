// Pieces of the cross-entropy shared by its own kernels and the epilogue of the product that makes the logits.
#pragma once
#include "zen_common.cuh"

namespace zen_xe {

constexpr float L2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// cap tanh(x / cap); *slope: its derivative 1 - tanh^2.  tanh.approx (relative error 2^-11) is no choice, whatever the type of the
// logits: the slope cancels near the cap (tanh 0.999: half of it would be noise), and fp32 logits have 13 more bits than it gives.
//  * fp32 logits: tanhf of the quotient, as in softcap_kernel: the loss is the loss of the logits that the model returns.
//  * 16-bit logits: from e = exp(-2 |x| / cap), tanh = (1 - e) / (1 + e) and slope = 4 e / (1 + e)^2, without cancellation at the
//    cap and within 3e-7 of tanh everywhere (2048 x 256 000 bf16 logits, both passes: 797 us; with tanhf 1 353, uncapped 503).
template <typename T>
__device__ __forceinline__ float xent_cap_value(float x, float cap, float k, float* slope) {
  if constexpr (sizeof(T) == 4) {
    const float t = tanhf(x / cap);
    *slope = 1.f - t * t;
    return cap * t;
  } else {
    const float e = ex2_fast(-fabsf(x) * k);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    *slope = 4.f * e * (r * r);
    return copysignf(cap * ((1.f - e) * r), x);
  }
}
template <typename T, bool CAP>
__device__ __forceinline__ float xent_cap(float x, float cap, float k, float* slope = nullptr) {
  if (!CAP) return x;
  float d;
  const float y = xent_cap_value<T>(x, cap, k, &d);
  if (slope) *slope = d;
  return y;
}

}  // namespace zen_xe
