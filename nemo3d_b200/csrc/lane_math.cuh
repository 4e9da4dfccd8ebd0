// Device helpers shared by the lane-per-(atom, spin) H*x kernels (spmv_ring.cu,
// spmv_pen.cu): complex multiply-adds, and explicitly rounded products for
// epilogues that several launch shapes must round identically.
#pragma once

namespace tbgpu {
namespace lanemath {

template <typename V> struct RealOf;
template <> struct RealOf<double2> { using T = double; };
template <> struct RealOf<float2> { using T = float; };

template <typename T, typename V>
__device__ __forceinline__ void cfma(V &acc, T h, V x) {
  acc.x = fma(h, x.x, acc.x);
  acc.y = fma(h, x.y, acc.y);
}
// acc += (i * lam) * x
template <typename T, typename V>
__device__ __forceinline__ void cfma_im(V &acc, T lam, V x) {
  acc.x = fma(-lam, x.y, acc.x);
  acc.y = fma(lam, x.x, acc.y);
}

// products that are never contracted into an FMA, so that every launch
// shape rounds the epilogue the same way
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

}  // namespace lanemath
}  // namespace tbgpu
