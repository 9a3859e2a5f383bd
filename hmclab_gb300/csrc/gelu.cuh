// GELU(z) = z Phi(z): first and second derivatives Phi(z) + z phi(z) and
// phi(z) (2 - z^2), with Phi(z) = erfc(-z / sqrt 2) / 2, which stays accurate in
// the negative tail (1 + erf cancels there in FP32).
#pragma once

namespace hmc {
namespace pot {

__device__ __forceinline__ float normal_pdf(float z) { return 0.39894228040143268f * __expf(-0.5f * z * z); }
__device__ __forceinline__ float gelu_d1(float z) {
  return 0.5f * erfcf(-z * 0.70710678118654752f) + z * normal_pdf(z);
}
__device__ __forceinline__ float gelu_d2(float z) { return normal_pdf(z) * (2.f - z * z); }

}  // namespace pot
}  // namespace hmc
