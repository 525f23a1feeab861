// The gate activations the epilogues implement, as compile-time variants (ids as in the C ABI), and
// the status codes a kernel can leave.
#pragma once
#include <cuda_runtime.h>

namespace moe {

enum Act { ACT_SILU = 0, ACT_GELU = 1, ACT_RELU = 2, ACT_SIGMOID = 3, ACT_TANH = 4 };

// Status codes a kernel can leave in the status word (0 = fine).
enum DevStatus { ST_OK = 0, ST_WAIT_TIMEOUT = 1, ST_BAD_EXPERT = 2 };

template <int ACT>
__device__ __forceinline__ float act_f(float g) {
  if constexpr (ACT == ACT_SILU) return __fdividef(g, 1.f + __expf(-g));
  if constexpr (ACT == ACT_GELU) return 0.5f * g * (1.f + erff(g * 0.7071067811865476f));
  if constexpr (ACT == ACT_RELU) return fmaxf(g, 0.f);
  if constexpr (ACT == ACT_SIGMOID) return __fdividef(1.f, 1.f + __expf(-g));
  return __fdividef(2.f, 1.f + __expf(-2.f * g)) - 1.f;
}
// (act(g), act'(g)) together: the backward needs both and they share the transcendental.
template <int ACT>
__device__ __forceinline__ void act_fd(float g, float& a, float& d) {
  if constexpr (ACT == ACT_SILU) {
    const float s = __fdividef(1.f, 1.f + __expf(-g));
    a = g * s;
    d = s * (1.f + g * (1.f - s));
  } else if constexpr (ACT == ACT_GELU) {
    const float cdf = 0.5f * (1.f + erff(g * 0.7071067811865476f));
    a = g * cdf;
    d = cdf + g * 0.3989422804014327f * __expf(-0.5f * g * g);
  } else if constexpr (ACT == ACT_RELU) {
    a = fmaxf(g, 0.f);
    d = g > 0.f ? 1.f : 0.f;
  } else if constexpr (ACT == ACT_SIGMOID) {
    a = __fdividef(1.f, 1.f + __expf(-g));
    d = a * (1.f - a);
  } else {
    a = __fdividef(2.f, 1.f + __expf(-2.f * g)) - 1.f;
    d = 1.f - a * a;
  }
}

}  // namespace moe
