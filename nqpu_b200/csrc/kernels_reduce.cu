// FP64 reductions over the statevector: all <Z_q> in one pass, inner products
// (fidelity), Pauli-string expectations and shot sampling.
//
// Reference semantics: QuantumState::expectation_z / fidelity /
// expectation_pauli_string / sample (R/lib.rs:388-560) and the C FFI's
// expectation_z / sample (c_ffi.rs:576-620).  The reference runs each of these
// as a serial loop per qubit or per term; here every reduction is one coalesced
// pass with FP64 accumulation: per-thread Kahan sums, warp-shuffle trees, and a
// final single-block FP64 combine, so results are deterministic for a given
// state and launch shape.  Pauli sums are in kernels_pauli.cu.
#include "reduce_device.cuh"

namespace nqpu {

// out[v] = sum over the blocks of part[v * nblk + b]: one warp per value, fixed
// order.  Values are strided by block so a warp's loads are coalesced.
__global__ void __launch_bounds__(1024)
    k_sum_rows(const double* __restrict__ part, int nvals, int nblk, double* __restrict__ out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int v = warp; v < nvals; v += int(blockDim.x >> 5)) {
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += part[size_t(v) * nblk + b];
    s = warp_sum(s);
    if (lane == 0) out[v] = s;
  }
}

cudaError_t launch_sum_rows(const double* part, int nvals, int nblk, double* out, cudaStream_t s) {
  k_sum_rows<<<1, 32 * std::min(nvals, 32), 0, s>>>(part, nvals, nblk, out);
  return cudaGetLastError();
}

// ---- all <Z_q> --------------------------------------------------------------
// A warp's work unit is a chunk of 32 lanes x 8 vectors (kZsChunkVecs).  Vector
// index bits 0..4 are lanes, 5..7 the thread's vectors, 8.. the chunk number.
// Per chunk a thread sums its 8 probabilities in a tree that also yields the
// sums over each of its three vector bits; only those five sums go through the
// compensated accumulators.  Lane b of the warp accumulates the chunk totals
// whose chunk bit b is set, so no per-segment array goes through memory and the
// final step adds (n + 1) rows of one value per block.
//
// Bound: HBM (the state is read once), FP64 issue close behind: 11 FP64
// operations per 128-bit vector here.  The earlier form took 22 (a compensated
// add per vector bit and vector), wrote one total per 4096 vectors and folded
// those in one block, which alone cost about 30 us of the 38 us of a 10-qubit
// call.  Measured (a call): 10 qubits complex64 37 -> 18 us, 20 qubits complex128
// 50 -> 28, 25 qubits complex64 (256 MB, 41 us at the copy rate) 98 -> 64.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
    k_zsums(const Real* __restrict__ amp, int n, uint64_t nchunks, double* __restrict__ part,
            double* __restrict__ out) {
  using V = typename Tr<Real>::V;
  constexpr int VB = Tr<Real>::kVecBit;
  constexpr int NV = int(kZsChunkVecs / 32);
  static_assert(NV == 8, "the tree below sums 8 vectors");
  const uint64_t nvec = (1ull << n) >> VB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  KSum tot, b0, j0, j1, j2, hi;
  const V* vp = reinterpret_cast<const V*>(amp);
  const uint64_t nwarps = uint64_t(gridDim.x) * kRedWarps;
  for (uint64_t ch = uint64_t(blockIdx.x) * kRedWarps + warp; ch < nchunks; ch += nwarps) {
    const uint64_t vb = ch * kZsChunkVecs + lane;
    V v[NV];
    if (vb - lane + kZsChunkVecs <= nvec) {
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = __ldcs(vp + vb + 32 * j);
    } else {  // a state of less than one chunk
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        v[j] = V{};
        if (vb + 32 * j < nvec) v[j] = __ldcs(vp + vb + 32 * j);
      }
    }
    double p[NV], odd = 0.0;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      double q[2];
      vec_probs<Real>(v[j], q);
      p[j] = q[0];
      if (VB == 1) {
        p[j] += q[1];
        odd += q[1];
      }
    }
    const double s01 = p[0] + p[1], s23 = p[2] + p[3], s45 = p[4] + p[5], s67 = p[6] + p[7];
    const double top = s45 + s67, t = (s01 + s23) + top;
    tot.add(t);
    if (VB == 1) b0.add(odd);
    j0.add((p[1] + p[3]) + (p[5] + p[7]));
    j1.add(s23 + s67);
    j2.add(top);
    const double w = warp_sum(t);
    if ((ch >> lane) & 1) hi.add(w);
  }
  // row v of the block: 0 total, 1 + q the sum over amplitudes with bit q set
  __shared__ double red[kRedWarps][kMaxQubits + 2];
  const double t = tot.s;
  double vals[6 + 5] = {t, b0.s, j0.s, j1.s, j2.s, 0.0};
#pragma unroll
  for (int b = 0; b < 5; ++b) vals[5 + b] = ((lane >> b) & 1) ? t : 0.0;
#pragma unroll
  for (int i = 0; i < 10; ++i) vals[i] = warp_sum(vals[i]);
  if (lane == 0) {
    red[warp][0] = vals[0];
    if (VB == 1) red[warp][1] = vals[1];
#pragma unroll
    for (int b = 0; b < 5; ++b) red[warp][1 + VB + b] = vals[5 + b];
#pragma unroll
    for (int b = 0; b < 3; ++b) red[warp][1 + VB + 5 + b] = vals[2 + b];
  }
  // chunk bits: qubits VB + 8 .. n - 1 (kMaxQubits of them at most)
  if (VB + 8 + lane < n) red[warp][1 + VB + 8 + lane] = hi.s;
  __syncthreads();
  if (tid <= n) {
    double s = 0.0;
    for (int w = 0; w < kRedWarps; ++w) s += red[w][tid];
    if (gridDim.x == 1) out[tid] = s;
    else part[size_t(tid) * gridDim.x + blockIdx.x] = s;
  }
}
static_assert(1 + 1 + 8 <= kMaxQubits + 2, "the chunk's own bits fit the row");

size_t reduce_scratch_bytes(int n) {
  size_t zs = sizeof(double) * zsums_scratch_doubles(n);
  size_t samp = sizeof(double) * (2 * ((1ull << n) / 4096 + 2) + 64);
  size_t inner = sizeof(double) * (2 * 4096 + 64);
  return std::max(zs, std::max(samp, inner)) + 4096;
}

template <typename Real>
static cudaError_t zsums_t(const Real* amp, int n, double* scratch, double* out, cudaStream_t s,
                           int num_sms) {
  const uint64_t nvec = (1ull << n) >> Tr<Real>::kVecBit;
  const uint64_t nchunks = std::max<uint64_t>(1, (nvec + kZsChunkVecs - 1) / kZsChunkVecs);
  // Up to four chunks per warp one block does it all (the second launch costs
  // about as much as three more chunks per warp); otherwise at least one chunk
  // per warp, at most three blocks per SM (96 KB of loads in flight per SM).
  uint64_t nblk = nchunks <= 4 * kRedWarps ? 1 : (nchunks + kRedWarps - 1) / kRedWarps;
  nblk = std::min<uint64_t>(nblk, std::min<uint64_t>(uint64_t(num_sms) * 3, kZsMaxBlocks));
  k_zsums<Real><<<unsigned(nblk), kRedThreads, 0, s>>>(amp, n, nchunks, scratch, out);
  if (nblk > 1) return launch_sum_rows(scratch, n + 1, int(nblk), out, s);
  return cudaGetLastError();
}

cudaError_t launch_zsums(DType dt, const void* amp, int n, double* scratch, double* out,
                         cudaStream_t s, int num_sms) {
  if (dt == DType::C64) return zsums_t<float>(static_cast<const float*>(amp), n, scratch, out, s, num_sms);
  return zsums_t<double>(static_cast<const double*>(amp), n, scratch, out, s, num_sms);
}

// ---- inner product ----------------------------------------------------------
// Two consecutive amplitudes of either precision in FP64.
__device__ __forceinline__ void load_pair(const float* p, uint64_t pair, double* v) {
  const float4 x = __ldcs(reinterpret_cast<const float4*>(p) + pair);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load_pair(const double* p, uint64_t pair, double* v) {
  const double2 x = __ldcs(reinterpret_cast<const double2*>(p) + 2 * pair);
  const double2 y = __ldcs(reinterpret_cast<const double2*>(p) + 2 * pair + 1);
  v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}

// Bound: HBM (both states are read once).  Four pairs of amplitudes per state
// in flight per thread as 128-bit loads; the eight products of a step are
// summed plainly and go through the compensated accumulators as one value.
// Measured (a call): 25 qubits complex64 (512 MB) 111 -> 100 us, 20 qubits
// complex128 36 -> 26, 10 qubits 24 -> 17.
template <typename RA, typename RB>
__global__ void __launch_bounds__(kRedThreads)
    k_inner(const RA* __restrict__ a, const RB* __restrict__ b, uint64_t npairs,
            double* __restrict__ part, double* __restrict__ out) {
  KSum re, im;
  const uint64_t stride = uint64_t(gridDim.x) * kRedThreads;
  uint64_t i = uint64_t(blockIdx.x) * kRedThreads + threadIdx.x;
  auto step = [&](const double* x, const double* y, double& r, double& m) {
    r += (x[0] * y[0] + x[1] * y[1]) + (x[2] * y[2] + x[3] * y[3]);
    m += (x[0] * y[1] - x[1] * y[0]) + (x[2] * y[3] - x[3] * y[2]);
  };
  for (; i + 3 * stride < npairs; i += 4 * stride) {
    double x[4][4], y[4][4], r = 0.0, m = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      load_pair(a, i + k * stride, x[k]);
      load_pair(b, i + k * stride, y[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) step(x[k], y[k], r, m);
    re.add(r);
    im.add(m);
  }
  for (; i < npairs; i += stride) {
    double x[4], y[4], r = 0.0, m = 0.0;
    load_pair(a, i, x);
    load_pair(b, i, y);
    step(x, y, r, m);
    re.add(r);
    im.add(m);
  }
  __shared__ double sh[2][kRedWarps];
  const double r = warp_sum(re.s), m = warp_sum(im.s);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sh[0][warp] = r; sh[1][warp] = m; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int w = 0; w < kRedWarps; ++w) t += sh[threadIdx.x][w];
    if (gridDim.x == 1) out[threadIdx.x] = t;
    else part[size_t(threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
}

cudaError_t launch_inner(DType dta, const void* a, DType dtb, const void* b, int n, double* scratch,
                         double* out, cudaStream_t s, int num_sms) {
  const uint64_t npairs = (1ull << n) >> 1;
  // one block up to 8 pairs per thread, else at least 4 per thread (one step)
  uint64_t nblk = npairs <= 8 * kRedThreads ? 1 : (npairs + 4 * kRedThreads - 1) / (4 * kRedThreads);
  nblk = std::min<uint64_t>(nblk, std::min<uint64_t>(uint64_t(num_sms) * 4, 4096));
  const unsigned g = unsigned(nblk);
  if (dta == DType::C64 && dtb == DType::C64)
    k_inner<float, float><<<g, kRedThreads, 0, s>>>(static_cast<const float*>(a), static_cast<const float*>(b), npairs, scratch, out);
  else if (dta == DType::C64)
    k_inner<float, double><<<g, kRedThreads, 0, s>>>(static_cast<const float*>(a), static_cast<const double*>(b), npairs, scratch, out);
  else if (dtb == DType::C64)
    k_inner<double, float><<<g, kRedThreads, 0, s>>>(static_cast<const double*>(a), static_cast<const float*>(b), npairs, scratch, out);
  else
    k_inner<double, double><<<g, kRedThreads, 0, s>>>(static_cast<const double*>(a), static_cast<const double*>(b), npairs, scratch, out);
  if (g > 1) return launch_sum_rows(scratch, 2, int(g), out, s);
  return cudaGetLastError();
}

// ---- Pauli string expectation (R/lib.rs:465) --------------------------------
// coeff(i) = i^ny * (-1)^popcount(i & zmask); j = i ^ xmask;
// result = sum_i Re(conj(a_i) * coeff(i) * a_j).
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
    k_pauli(const Real* __restrict__ amp, uint64_t dim, uint64_t xmask, uint64_t zmask, int ny,
            double* __restrict__ part) {
  KSum acc;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < dim; i += stride) {
    const uint64_t j = i ^ xmask;
    const double ar = amp[2 * i], ai = amp[2 * i + 1];
    const double br = amp[2 * j], bi = amp[2 * j + 1];
    // c = i^ny * sign
    double cr, ci;
    switch (ny & 3) {
      case 0: cr = 1; ci = 0; break;
      case 1: cr = 0; ci = 1; break;
      case 2: cr = -1; ci = 0; break;
      default: cr = 0; ci = -1; break;
    }
    if (__popcll(i & zmask) & 1) { cr = -cr; ci = -ci; }
    const double pr = cr * br - ci * bi;
    const double pi = cr * bi + ci * br;
    acc.add(ar * pr + ai * pi);
  }
  __shared__ double sh[kRedThreads / 32];
  double r = warp_sum(acc.s);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0;
    for (int w = 0; w < kRedThreads / 32; ++w) sr += sh[w];
    part[blockIdx.x] = sr;
  }
}

cudaError_t launch_pauli(DType dt, const void* amp, int n, uint64_t xmask, uint64_t zmask,
                         uint64_t ymask, double* scratch, double* out, cudaStream_t s,
                         int num_sms) {
  const uint64_t dim = 1ull << n;
  int nblk = int(std::min<uint64_t>((dim + kRedThreads - 1) / kRedThreads, uint64_t(num_sms) * 8));
  nblk = std::max(1, std::min(nblk, 4096));
  const int ny = __builtin_popcountll(ymask);
  if (dt == DType::C64)
    k_pauli<float><<<nblk, kRedThreads, 0, s>>>(static_cast<const float*>(amp), dim, xmask, zmask, ny, scratch);
  else
    k_pauli<double><<<nblk, kRedThreads, 0, s>>>(static_cast<const double*>(amp), dim, xmask, zmask, ny, scratch);
  return launch_sum_rows(scratch, 1, nblk, out, s);
}

// ---- sampling ---------------------------------------------------------------
constexpr int kSampSegBits = 12;  // 4096 amplitudes per CDF segment

// Segment sums.  Bound: HBM.  A full segment is 256 threads x 16 amplitudes, all
// of a thread's 128-bit loads in flight at once (complex64 8, complex128 16);
// the scalar form moved one 4- or 8-byte load per step.
template <typename Real>
__global__ void __launch_bounds__(kRedThreads)
    k_seg_probs(const Real* __restrict__ amp, uint64_t nseg, int segbits, double* __restrict__ seg_sum) {
  using V = typename Tr<Real>::V;
  constexpr int VB = Tr<Real>::kVecBit;
  constexpr int NV = (1 << (kSampSegBits - VB)) / kRedThreads;
  __shared__ double sh[kRedWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t segvec = (1ull << segbits) >> VB;
  const V* vp = reinterpret_cast<const V*>(amp);
  for (uint64_t sg = blockIdx.x; sg < nseg; sg += gridDim.x) {
    V v[NV];
    const uint64_t b = sg * segvec;
    if (segvec == uint64_t(NV) * kRedThreads) {
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = __ldcs(vp + b + threadIdx.x + j * kRedThreads);
    } else {  // a state of less than one segment
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const uint64_t k = threadIdx.x + uint64_t(j) * kRedThreads;
        v[j] = V{};
        if (k < segvec) v[j] = __ldg(vp + b + k);
      }
    }
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      double p[2];
      vec_probs<Real>(v[j], p);
      acc += VB == 1 ? p[0] + p[1] : p[0];
    }
    acc = warp_sum(acc);
    if (lane == 0) sh[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int w = 0; w < kRedWarps; ++w) t += sh[w];
      seg_sum[sg] = t;
    }
    __syncthreads();
  }
}

// Inclusive scan of seg_sum into seg_incl (single block, FP64, deterministic):
// tiles of 4 consecutive values per thread with a running carry, so every load
// is coalesced and a state of 2^24 amplitudes is one tile.
__global__ void __launch_bounds__(1024)
    k_seg_scan(const double* __restrict__ seg_sum, uint64_t nseg, double* __restrict__ seg_incl) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double carry = 0.0;
  for (uint64_t t0 = 0; t0 < nseg; t0 += 4096) {
    const uint64_t b = t0 + uint64_t(threadIdx.x) * 4;
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = b + k < nseg ? seg_sum[b + k] : 0.0;
    v[1] += v[0];
    v[2] += v[1];
    v[3] += v[2];
    double sc = v[3];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, sc, o);
      if (lane >= o) sc += t;
    }
    if (lane == 31) sh[warp] = sc;
    __syncthreads();
    double ws = sh[lane];  // every warp scans the 32 warp totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += t;
    }
    const double before_warp = __shfl_sync(0xffffffffu, ws, warp ? warp - 1 : 0);
    const double before_lane = __shfl_up_sync(0xffffffffu, sc, 1);
    double base = carry;
    if (warp) base += before_warp;
    if (lane) base += before_lane;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (b + k < nseg) seg_incl[b + k] = base + v[k];
    carry += __shfl_sync(0xffffffffu, ws, 31);
    __syncthreads();  // sh is rewritten by the next tile
  }
}

// One warp per shot, for few shots.  In a segment a step covers 32 lanes x 8 vectors: each lane
// loads 8 consecutive vectors at once, sums its probabilities serially, and the
// warp scans the 32 lane totals; the lane whose range holds r then picks the
// amplitude from its own prefix.  A segment is 8 (complex64) or 16 (complex128)
// dependent steps instead of 128 of one amplitude per lane.  Measured (1024
// shots, the whole call): 25 qubits complex64 202 -> 97 us, 20 qubits complex128
// 99 -> 59, 10 qubits 56 -> 44.
template <typename Real>
__global__ void __launch_bounds__(256, 2)
    k_sample(const Real* __restrict__ amp, uint64_t dim, int segbits, uint64_t nseg,
             const double* __restrict__ seg_sum, const double* __restrict__ seg_incl,
             const double* __restrict__ u, uint32_t shots, uint64_t* __restrict__ out) {
  using V = typename Tr<Real>::V;
  constexpr int VB = Tr<Real>::kVecBit;
  constexpr int NV = 8, NP = NV << VB;  // vectors and amplitudes of a lane's step
  const V* vp = reinterpret_cast<const V*>(amp);
  const int lane = threadIdx.x & 31;
  const uint64_t warp_id = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  const uint64_t nvec = dim >> VB;
  for (uint64_t sh = warp_id; sh < shots; sh += nwarps) {
    const double r = u[sh];
    // first segment whose inclusive prefix exceeds r
    uint64_t lo = 0, hi = nseg;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (seg_incl[mid] > r) hi = mid; else lo = mid + 1;
    }
    uint64_t result = dim - 1;
    bool found = false;
    for (uint64_t sg = lo; sg < nseg && !found; ++sg) {
      double run = seg_incl[sg] - seg_sum[sg];
      const uint64_t v0 = (sg << segbits) >> VB;
      const uint64_t seg_end = v0 + ((1ull << segbits) >> VB);
      const uint64_t v1 = seg_end < nvec ? seg_end : nvec;
      for (uint64_t b = v0; b < v1; b += 32 * NV) {
        const uint64_t k = b + uint64_t(lane) * NV;
        V v[NV];
        if (b + 32 * NV <= v1) {
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = __ldg(vp + k + j);
        } else {
#pragma unroll
          for (int j = 0; j < NV; ++j) {
            v[j] = V{};
            if (k + j < v1) v[j] = __ldg(vp + k + j);
          }
        }
        double p[NP];  // inclusive prefix within the lane
#pragma unroll
        for (int j = 0; j < NV; ++j) vec_probs<Real>(v[j], p + (j << VB));
#pragma unroll
        for (int j = 1; j < NP; ++j) p[j] += p[j - 1];
        double sc = p[NP - 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double t = __shfl_up_sync(0xffffffffu, sc, o);
          if (lane >= o) sc += t;
        }
        const double excl = __shfl_up_sync(0xffffffffu, sc, 1);
        const double base = lane ? run + excl : run;
        const unsigned hit = __ballot_sync(0xffffffffu, k < v1 && r < base + p[NP - 1]);
        if (hit) {
          const int src = __ffs(hit) - 1;
          int first = NP - 1;
#pragma unroll
          for (int j = NP - 2; j >= 0; --j)
            if (r < base + p[j]) first = j;
          const uint64_t i = (k << VB) + unsigned(first);
          result = __shfl_sync(0xffffffffu, i, src);
          found = true;
          break;
        }
        run += __shfl_sync(0xffffffffu, sc, 31);
      }
    }
    if (lane == 0) out[sh] = result < dim ? result : dim - 1;
  }
}

// The same for many shots, where the loads of the form above count (eight consecutive
// vectors per lane: every load touches 32 lines).  A step covers NV rows of 32
// vectors, a vector per lane and row.  A step that r lies beyond costs one sum over
// the warp; in the one that holds r every row is scanned, all rows at once, and the
// first amplitude whose prefix exceeds r is taken.  Without SKIP (states of a few rows)
// every step is scanned.
// Measured (100000 shots, the whole call; one amplitude per lane and step, the form
// above, this one):
//   13 qubits   complex64   877  705  379 us     complex128   860 1185  391
//   25 qubits   complex64  1126  713  480        complex128  1142 1197  534
template <typename Real, int NV, bool SKIP>
__global__ void __launch_bounds__(256, 2)
    k_sample_rows(const Real* __restrict__ amp, uint64_t dim, int segbits, uint64_t nseg,
             const double* __restrict__ seg_sum, const double* __restrict__ seg_incl,
             const double* __restrict__ u, uint32_t shots, uint64_t* __restrict__ out) {
  using V = typename Tr<Real>::V;
  constexpr int VB = Tr<Real>::kVecBit;
  const V* vp = reinterpret_cast<const V*>(amp);
  const int lane = threadIdx.x & 31;
  const uint64_t warp_id = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  const uint64_t nvec = dim >> VB;
  for (uint64_t sh = warp_id; sh < shots; sh += nwarps) {
    const double r = u[sh];
    // first segment whose inclusive prefix exceeds r
    uint64_t lo = 0, hi = nseg;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (seg_incl[mid] > r) hi = mid; else lo = mid + 1;
    }
    uint64_t result = dim - 1;
    bool found = false;
    for (uint64_t sg = lo; sg < nseg && !found; ++sg) {
      double run = seg_incl[sg] - seg_sum[sg];
      const uint64_t v0 = (sg << segbits) >> VB;
      const uint64_t seg_end = v0 + ((1ull << segbits) >> VB);
      const uint64_t v1 = seg_end < nvec ? seg_end : nvec;
      for (uint64_t b = v0; b < v1 && !found; b += 32 * NV) {
        const uint64_t k = b + lane;
        V v[NV];
        if (b + 32 * NV <= v1) {
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = __ldg(vp + k + 32 * j);
        } else {
#pragma unroll
          for (int j = 0; j < NV; ++j) {
            v[j] = V{};
            if (k + 32 * j < v1) v[j] = __ldg(vp + k + 32 * j);
          }
        }
        double p0[NV], sc[NV], t = 0.0;  // the vector's first amplitude, all of it
        uint32_t some = 0, later = 0;    // bit j: row j's vector, its second amplitude is not 0
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          double p[2];
          vec_probs<Real>(v[j], p);
          p0[j] = p[0];
          sc[j] = VB == 1 ? p[0] + p[1] : p[0];
          t += sc[j];
          some |= uint32_t(sc[j] > 0.0) << j;
          if (VB == 1) later |= uint32_t(p[1] > 0.0) << j;
        }
        if (SKIP) {
          t = warp_sum(t);
          if (!(r < run + t)) {
            run += t;
            continue;
          }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
          for (int j = 0; j < NV; ++j) {
            const double x = __shfl_up_sync(0xffffffffu, sc[j], o);
            if (lane >= o) sc[j] += x;
          }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          // (only what has a probability: two lanes' prefixes may differ by a rounding)
          const unsigned hit = __ballot_sync(0xffffffffu, ((some >> j) & 1u) && r < run + sc[j]);
          if (hit && !found) {
            const double excl = __shfl_up_sync(0xffffffffu, sc[j], 1);
            const bool second = ((later >> j) & 1u) && !(r < run + (lane ? excl : 0.0) + p0[j]);
            result = __shfl_sync(0xffffffffu, ((k + 32 * j) << VB) + (second ? 1 : 0), __ffs(hit) - 1);
            found = true;
          }
          run += __shfl_sync(0xffffffffu, sc[j], 31);
        }
      }
    }
    if (lane == 0) out[sh] = result < dim ? result : dim - 1;
  }
}

// From this many shots on by rows: below, a call's latency counts and either form
// takes about as long.
constexpr uint32_t kRowShots = 2017;

template <typename Real>
static void sample_t(const Real* amp, uint64_t dim, int segbits, uint64_t nseg, const double* seg_sum,
                     const double* seg_incl, const double* u, uint32_t shots, uint64_t* out, int grid, cudaStream_t s) {
  auto go = [&](auto kernel) {
    kernel<<<grid, 256, 0, s>>>(amp, dim, segbits, nseg, seg_sum, seg_incl, u, shots, out);
  };
  const uint64_t rows = (dim >> Tr<Real>::kVecBit) >> 5;
  if (shots < kRowShots) go(k_sample<Real>);
  else if (rows <= 4) go(k_sample_rows<Real, 1, false>);
  else if (rows <= 8) go(k_sample_rows<Real, 4, true>);
  else go(k_sample_rows<Real, 8, true>);
}

cudaError_t launch_sample(DType dt, const void* amp, int n, const double* d_uniforms,
                          uint32_t shots, double* scratch, uint64_t* d_out, cudaStream_t s,
                          int num_sms) {
  const uint64_t dim = 1ull << n;
  const int segbits = n < kSampSegBits ? n : kSampSegBits;
  const uint64_t nseg = dim >> segbits;
  double* seg_sum = scratch;
  double* seg_incl = scratch + nseg + 1;
  const int g1 = int(std::min<uint64_t>(nseg, uint64_t(num_sms) * 6));
  if (dt == DType::C64)
    k_seg_probs<float><<<g1, kRedThreads, 0, s>>>(static_cast<const float*>(amp), nseg, segbits, seg_sum);
  else
    k_seg_probs<double><<<g1, kRedThreads, 0, s>>>(static_cast<const double*>(amp), nseg, segbits, seg_sum);
  k_seg_scan<<<1, 1024, 0, s>>>(seg_sum, nseg, seg_incl);
  if (shots == 0) return cudaGetLastError();
  const uint64_t warps = shots;
  const int g2 = int(std::max<uint64_t>(1, std::min<uint64_t>((warps * 32 + 255) / 256, uint64_t(num_sms) * 8)));
  if (dt == DType::C64)
    sample_t(static_cast<const float*>(amp), dim, segbits, nseg, seg_sum, seg_incl, d_uniforms, shots, d_out, g2, s);
  else
    sample_t(static_cast<const double*>(amp), dim, segbits, nseg, seg_sum, seg_incl, d_uniforms, shots, d_out, g2, s);
  return cudaGetLastError();
}

}  // namespace nqpu
