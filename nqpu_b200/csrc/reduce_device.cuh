// Device code shared by the FP64 reduction kernels.  Included by .cu files only.
#pragma once
#include "kernels.h"
#include "sv_device.cuh"

namespace nqpu {

// Compensated (Kahan) accumulator.
struct KSum {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double x) {
    double y = x - c;
    double t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int kRedThreads = 256;
constexpr int kRedWarps = kRedThreads / 32;

template <typename Real>
__device__ __forceinline__ void vec_probs(const typename Tr<Real>::V& v, double* p);
template <>
__device__ __forceinline__ void vec_probs<float>(const float4& v, double* p) {
  p[0] = double(v.x) * double(v.x) + double(v.y) * double(v.y);
  p[1] = double(v.z) * double(v.z) + double(v.w) * double(v.w);
}
template <>
__device__ __forceinline__ void vec_probs<double>(const double2& v, double* p) {
  p[0] = v.x * v.x + v.y * v.y;
}

}  // namespace nqpu
