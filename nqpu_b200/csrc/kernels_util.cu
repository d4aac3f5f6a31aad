// Elementwise state kernels: basis-state init (QuantumState::new / reset,
// R/lib.rs:331 and c_ffi.rs:233), scaling/renormalisation, measurement
// collapse (c_ffi.rs:537-566, GateOperations::reset_qubit R/lib.rs:1705),
// probabilities (R/lib.rs:354) and dtype conversion.
#include "sv_device.cuh"
#include "kernels.h"

namespace nqpu {

static unsigned ew_grid(uint64_t items, int num_sms) {
  const uint64_t max_blocks = uint64_t(num_sms) * 8;
  uint64_t need = (items + 255) / 256;
  if (need < 1) need = 1;
  return unsigned(need < max_blocks ? need : max_blocks);
}

template <typename Real>
__global__ void k_set_basis(Real* __restrict__ amp, uint64_t dim2, uint64_t index) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim2; i += stride)
    amp[i] = (i == 2 * index) ? Real(1) : Real(0);
}

template <typename Real>
__global__ void k_scale(Real* __restrict__ amp, uint64_t dim2, Real f) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim2; i += stride)
    amp[i] *= f;
}

template <typename Real>
__global__ void k_collapse(Real* __restrict__ amp, uint64_t dim, int q, int keep, Real f) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim; i += stride) {
    const bool k = int((i >> q) & 1) == keep;
    amp[2 * i] = k ? amp[2 * i] * f : Real(0);
    amp[2 * i + 1] = k ? amp[2 * i + 1] * f : Real(0);
  }
}

// Measurement collapse with the outcome decided on the device (c_ffi.rs:537-566):
// sums = launch_zsums' output, r the uniform draw; outcome 0 when r < prob(0).  The
// kept half is scaled to norm 1 and the other one zeroed; with `flip` outcome 1
// moves to the |0> half (OpenQASM reset).  Reads only the kept half.  result
// (device or pinned host memory, may be null): outcome, probability.
//
// The decision used to be the host's, a synchronisation and a launch gap of
// about 15 us per measurement; queued this way the measurements of a circuit
// run back to back.  Items are pairs of 128-bit vectors (complex64 qubit 0: one
// vector holds the pair).
template <typename Real>
__global__ void __launch_bounds__(256)
    k_measure_collapse(Real* __restrict__ amp, int n, int q, const double* __restrict__ sums, double r, int flip,
                       double* __restrict__ result) {
  using V = typename Tr<Real>::V;
  constexpr int VB = Tr<Real>::kVecBit;
  const double prob0 = sums[0] - sums[1 + q];  // sum over bit q == 0
  const double prob1 = 1.0 - prob0;            // c_ffi.rs:546
  const int out = r < prob0 ? 0 : 1;
  const double po = out == 0 ? prob0 : prob1;
  const Real f = Real(1.0 / sqrt(po));
  if (result && blockIdx.x == 0 && threadIdx.x == 0) {
    result[0] = double(out);
    result[1] = po;
  }
  const int to = flip ? 0 : out;  // the half that ends up with the amplitudes
  V* vp = reinterpret_cast<V*>(amp);
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  const uint64_t nvec = (1ull << n) >> VB;
  const uint64_t i0 = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if constexpr (VB == 1) {
    if (q == 0) {
      for (uint64_t i = i0; i < nvec; i += stride) {
        const float4 v = vp[i];
        const float x = (out ? v.z : v.x) * f, y = (out ? v.w : v.y) * f;
        vp[i] = to ? make_float4(0.f, 0.f, x, y) : make_float4(x, y, 0.f, 0.f);
      }
      return;
    }
  }
  const uint64_t bit = 1ull << (q - VB);
  for (uint64_t i = i0; i < nvec / 2; i += stride) {
    const uint64_t lo = insert_zero_bit(i, q - VB);
    V v = vp[lo | (out ? bit : 0)];
    v.x *= f;
    v.y *= f;
    if constexpr (VB == 1) { v.z *= f; v.w *= f; }
    vp[lo | (to ? bit : 0)] = v;
    vp[lo | (to ? 0 : bit)] = V{};
  }
}

template <typename Real>
__global__ void k_probs(const Real* __restrict__ amp, uint64_t dim, double* __restrict__ out) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim; i += stride) {
    const double r = amp[2 * i], m = amp[2 * i + 1];
    out[i] = r * r + m * m;
  }
}

template <typename RS, typename RD>
__global__ void k_convert(const RS* __restrict__ src, RD* __restrict__ dst, uint64_t dim2) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim2; i += stride)
    dst[i] = RD(src[i]);
}

cudaError_t launch_set_basis(DType dt, void* amp, int n, uint64_t index, cudaStream_t s, int num_sms) {
  const uint64_t dim2 = 2ull << n;
  if (dt == DType::C64) k_set_basis<float><<<ew_grid(dim2, num_sms), 256, 0, s>>>(static_cast<float*>(amp), dim2, index);
  else k_set_basis<double><<<ew_grid(dim2, num_sms), 256, 0, s>>>(static_cast<double*>(amp), dim2, index);
  return cudaGetLastError();
}

cudaError_t launch_scale(DType dt, void* amp, int n, double factor, cudaStream_t s, int num_sms) {
  const uint64_t dim2 = 2ull << n;
  if (dt == DType::C64) k_scale<float><<<ew_grid(dim2, num_sms), 256, 0, s>>>(static_cast<float*>(amp), dim2, float(factor));
  else k_scale<double><<<ew_grid(dim2, num_sms), 256, 0, s>>>(static_cast<double*>(amp), dim2, factor);
  return cudaGetLastError();
}

cudaError_t launch_collapse(DType dt, void* amp, int n, int q, int keep, double factor,
                            cudaStream_t s, int num_sms) {
  const uint64_t dim = 1ull << n;
  if (dt == DType::C64) k_collapse<float><<<ew_grid(dim, num_sms), 256, 0, s>>>(static_cast<float*>(amp), dim, q, keep, float(factor));
  else k_collapse<double><<<ew_grid(dim, num_sms), 256, 0, s>>>(static_cast<double*>(amp), dim, q, keep, factor);
  return cudaGetLastError();
}

cudaError_t launch_measure_collapse(DType dt, void* amp, int n, int q, const double* sums, double r, bool flip,
                                    double* result, cudaStream_t s, int num_sms) {
  const uint64_t items = std::max<uint64_t>(1, (1ull << n) >> 1);
  if (dt == DType::C64) k_measure_collapse<float><<<ew_grid(items, num_sms), 256, 0, s>>>(static_cast<float*>(amp), n, q, sums, r, flip, result);
  else k_measure_collapse<double><<<ew_grid(items, num_sms), 256, 0, s>>>(static_cast<double*>(amp), n, q, sums, r, flip, result);
  return cudaGetLastError();
}

cudaError_t launch_probabilities(DType dt, const void* amp, uint64_t count, double* out, cudaStream_t s, int num_sms) {
  const uint64_t dim = count;
  if (dt == DType::C64) k_probs<float><<<ew_grid(dim, num_sms), 256, 0, s>>>(static_cast<const float*>(amp), dim, out);
  else k_probs<double><<<ew_grid(dim, num_sms), 256, 0, s>>>(static_cast<const double*>(amp), dim, out);
  return cudaGetLastError();
}

cudaError_t launch_convert(DType sdt, const void* src, DType ddt, void* dst, uint64_t count, cudaStream_t s, int num_sms) {
  const uint64_t dim2 = 2ull * count;
  const unsigned g = ew_grid(dim2, num_sms);
  if (sdt == DType::C64 && ddt == DType::C128) k_convert<float, double><<<g, 256, 0, s>>>(static_cast<const float*>(src), static_cast<double*>(dst), dim2);
  else if (sdt == DType::C128 && ddt == DType::C64) k_convert<double, float><<<g, 256, 0, s>>>(static_cast<const double*>(src), static_cast<float*>(dst), dim2);
  else if (sdt == DType::C64) k_convert<float, float><<<g, 256, 0, s>>>(static_cast<const float*>(src), static_cast<float*>(dst), dim2);
  else k_convert<double, double><<<g, 256, 0, s>>>(static_cast<const double*>(src), static_cast<double*>(dst), dim2);
  return cudaGetLastError();
}

}  // namespace nqpu
