// The surrogate's activation and its derivative.
#pragma once

namespace ifdtd {
namespace nn {

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.f / (1.f + expf(-z));
  return s * (1.f + z * (1.f - s));
}

}  // namespace nn
}  // namespace ifdtd
