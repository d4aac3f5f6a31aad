// Tiled multi-gate pass kernel (the plain method's main path).
//
// One launch = one HBM pass over the state: each CTA streams tiles of 2^k
// amplitudes (k <= 13 for complex64, 12 for complex128: 64 KB) from HBM into
// shared memory with coalesced 128-bit loads, applies every gate the planner
// assigned to the pass, and streams the tile back.  Gates run in register
// stages: each thread gathers 16 vectors (32 complex64 / 16 complex128
// amplitudes) that differ in the stage's register bits, applies all of the
// stage's ops with fully unrolled register code, and scatters them back.
//
// Reference semantics: each op performs the same per-amplitude arithmetic as
// GateOperations (R/lib.rs:617-1735) — 2x2 rows a*x + b*y for dense 1q gates
// (apply_unitary_pair_indexed, R/lib.rs:634), 4x4 rows for u2 (R/lib.rs:1536),
// swaps for X/CNOT/SWAP (R/lib.rs:712/835/1207) and phases for diagonal gates —
// in the state's own precision.
//
// Shared-memory layout: vector u (16 B) lives at slot swz(u) = u ^ fold3(u>>3)
// so that the 8 lanes of a quarter-warp that the planner maps to vector bits of
// distinct residue mod 3 hit 8 distinct 16-byte bank groups.
#include <atomic>
#include "device_once.h"
#include "kernels.h"
#include "tile_device.cuh"

namespace nqpu {

// Dynamic shared memory: [tile buffer 0 | tile buffer 1 | hi_off table
// (2^(k-c) <= kHiOffEntries u64) | stage tables of the pass (kStageTabWords u32
// each) | the pass's program].
// WAY 0: the program stays in global memory (it does not fit); 1: it is in shared
// memory; 2: that, and the tile has all of KMAX bits.  Kernels of their own,
// because deciding it inside costs the stage loop spills (complex128 at 128
// registers: 20-qubit brickwork 398 us against 385; the forms apart spill 8 to 40
// bytes there, complex64 none but 76 where the program is in global memory).
// MINB = 1: one persistent CTA per SM; while the stages of tile i run on one
// buffer, the cp.async copies of tile i+1 stream into the other.  MINB > 1:
// MINB CTAs per SM with one buffer each hide each other's copies.  Each thread
// holds 16 vectors, so a CTA has 2^KMAX / (16 x amplitudes per vector) threads.
template <typename Real, int KMAX, int MINB, int WAY>
__global__ void __launch_bounds__(1 << (KMAX - Tr<Real>::kVecBit - 4), MINB)
    k_tile_pass(Real* __restrict__ amp, const __grid_constant__ PassRec P, const uint4* __restrict__ progs,
                uint32_t n_tiles, uint64_t out_mask, uint64_t step) {
  using T = Tr<Real>;
  using V = typename T::V;
  constexpr int VB = T::kVecBit;
  constexpr uint32_t kMaxVec = 1u << (KMAX - VB);
  constexpr int kThreads = int(kMaxVec) / kVecPerThread;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool kDoubleBuffer = (MINB == 1);
  V* buf0 = reinterpret_cast<V*>(smem_raw);
  V* buf1 = kDoubleBuffer ? buf0 + kMaxVec : buf0;
  uint64_t* hi_off = reinterpret_cast<uint64_t*>(smem_raw + (kDoubleBuffer ? 2 : 1) * sizeof(V) * kMaxVec);
  uint32_t* tabs = reinterpret_cast<uint32_t*>(hi_off + kHiOffEntries);
  const int tid = threadIdx.x;
  const int k = P.k, c = P.c;
  const uint32_t nvec = 1u << (k - VB);
  const int nhi = k - c;
  const int tab_words = (P.stage_end - P.stage_begin) * (kStageTabWords / 4);
  load_pass_prog(P, progs, WAY ? P.prog_words - tab_words : 0, reinterpret_cast<uint4*>(tabs));
  for (int h = tid; h < (1 << nhi); h += blockDim.x) {
    uint64_t off = 0;
    for (int j = 0; j < nhi; ++j)
      if ((h >> j) & 1) off |= 1ull << P.qhi[j];
    hi_off[h] = off;
  }
  const uint4* prog_s = reinterpret_cast<const uint4*>(tabs) + tab_words;
  const uint4* prog_g = progs + P.prog_begin + tab_words;
  cp_async_wait0();
  __syncthreads();
  // everything above read only the plan's tables: the previous pass of the
  // state may still be running up to here
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t lowmask = (1u << c) - 1u;
  using Copy = TileCopy<Real, KMAX>;
  const bool full = WAY == 2 || Copy::fits(P);

  // HBM -> shared, asynchronous (consecutive threads take consecutive vectors).
  auto issue_load = [&](uint64_t base, V* dst) {
    if (full) {
      Copy::each(amp, P, hi_off, base, [&](uint32_t slot, V* g) { cp_async16(dst + slot, g); });
      return;
    }
#pragma unroll 1
    for (uint32_t u = tid; u < nvec; u += kThreads) {
      const uint32_t t = u << VB;
      cp_async16(dst + swz(u), amp + 2 * (base + (t & lowmask) + hi_off[t >> c]));
    }
  };
  // the tile gridDim.x further on: an addition of `step`, the grid size laid out
  // over the qubits outside the tile, with the carries running over the gaps
  auto advance = [&](uint64_t base) { return ((base | ~out_mask) + step) & out_mask; };

  uint64_t base = tile_base(P, blockIdx.x);
  if (kDoubleBuffer) {
    if (blockIdx.x < n_tiles) issue_load(base, buf0);
    cp_async_commit();
  }
  for (uint32_t it = 0, tile = blockIdx.x; tile < n_tiles; ++it, tile += gridDim.x) {
    V* sv = (it & 1) ? buf1 : buf0;
    if (kDoubleBuffer) {
      if (tile + gridDim.x < n_tiles) issue_load(advance(base), (it & 1) ? buf0 : buf1);
    } else {
      issue_load(base, sv);  // single buffer: the other CTA on the SM hides the latency
    }
    cp_async_commit();
    if (kDoubleBuffer) cp_async_wait1();  // everything but the newest group (the prefetch) has landed
    else cp_async_wait0();
    __syncthreads();

    // lane j holds the bit of ext qubit j
    int lane = threadIdx.x & 31;
    asm volatile("" : "+r"(lane));  // worked out per tile: no registers held across the stages
    const uint32_t ext =
        __ballot_sync(0xffffffffu, lane < P.n_ext && ((base >> P.ext[lane]) & 1ull)) << k;

    constexpr bool kFew = sizeof(Real) == 8 && MINB > 1;
    if constexpr (WAY > 0) run_tile_stages<Real, kFew>(sv, P, tabs, prog_s, ext);
    else run_tile_stages<Real, kFew>(sv, P, tabs, prog_g, ext);

    // shared -> HBM
    if (full) {
      Copy::each(amp, P, hi_off, base, [&](uint32_t slot, V* g) { __stcs(g, sv[slot]); });
    } else {
#pragma unroll 1
      for (uint32_t u = tid; u < nvec; u += kThreads) {
        const uint32_t t = u << VB;
        __stcs(reinterpret_cast<V*>(amp + 2 * (base + (t & lowmask) + hi_off[t >> c])), sv[swz(u)]);
      }
    }
    __syncthreads();  // this buffer is refilled by the prefetch issued next iteration
    base = advance(base);
  }
}

// Largest tile (bits) per dtype: 64 KB of amplitudes.
template <typename Real>
constexpr int tile_kmax_full() { return sizeof(Real) == 4 ? 13 : 12; }

template <typename Real, int KMAX>
static size_t tile_smem_base(int minb) {
  using V = typename Tr<Real>::V;
  return (minb == 1 ? 2 : 1) * sizeof(V) * (size_t(1) << (KMAX - Tr<Real>::kVecBit)) +
         sizeof(uint64_t) * kHiOffEntries;
}
// Most dynamic shared memory of a CTA when MINB of them share an SM's 227 KB
// (1 KB each goes to the system, under 1 KB to the static arrays); enough for
// the tables of the longest pass.
template <typename Real, int KMAX>
static size_t tile_smem_max(int minb, int share_of) {
  const size_t need = tile_smem_base<Real, KMAX>(minb) + sizeof(uint32_t) * kMaxPassStages * kStageTabWords;
  const size_t share = size_t(227 * 1024) / size_t(share_of) - 2048;
  return std::max(need, share);
}

// CTA configuration of the tiled pass kernel per dtype (CTAs per SM):
//   1: one 64 KB-tile CTA per SM, double-buffered (cp.async prefetch of the next tile);
//   2: two 64 KB-tile CTAs per SM, one buffer each;
//   4: four CTAs per SM on 32 KB tiles (one tile bit fewer, half the threads):
//      more independent CTAs to overlap each other's barriers and copies, at
//      the price of more passes;
//   0: not set: chosen per plan and launch.
//     complex64: 4, or 2 for a plan on 13-bit tiles (build_tile_plan_for).
//     complex128: 1 while there is at most one tile per SM (no spills, matrices
//     in registers: a 13-qubit ansatz takes 72 us against 74; 8 qubits of 4x4s 95
//     against 122), else 2 (four warps per scheduler instead of two hide the
//     dependency waits: 25-qubit ansatz of 8 layers 5.1 against 6.6 ms, 20-qubit
//     brickwork 383 against 461 us; 4 takes 4.7 ms and 389 us, with 12 and 21
//     passes for 10 and 14: the better one on large states, which no rule here
//     separates yet).
static std::atomic<int> g_tile_minb[2];

void tile_config_set(DType dt, int minb) { g_tile_minb[dt == DType::C64 ? 0 : 1] = minb; }
int tile_config_get(DType dt) { return g_tile_minb[dt == DType::C64 ? 0 : 1]; }

template <typename Real, int KMAX, int MINB, int WAY>
cudaError_t launch_tile_pass_cfg(Real* amp, const PassRec& host_pass, const ProgWord* d_prog,
                                 cudaStream_t stream, int num_sms) {
  // a plan built for larger tiles than this kernel holds must not run on it,
  // nor one whose tables exceed the shared-memory copies
  if (host_pass.k > KMAX || host_pass.k < 1 || host_pass.k - host_pass.c > kHiOffBits ||
      host_pass.stage_end - host_pass.stage_begin > kMaxPassStages)
    return cudaErrorInvalidValue;
  auto kern = k_tile_pass<Real, KMAX, MINB, WAY>;
  constexpr int kThreads = (1 << (KMAX - Tr<Real>::kVecBit)) / kVecPerThread;
  // shared memory of this launch: the tile buffer(s), the high-offset table, the
  // stage tables of this pass and, where it fits beside them in MINB CTAs per
  // SM, its program (a single-tile CTA would wait for each op's first read
  // from L2 otherwise)
  // Fewer tiles than the GPU takes at once leave more of the SM's to each CTA (96
  // 4x4 gates on 8 qubits: their program from global memory 201 us, from here 171).
  const uint32_t n_tiles = 1u << host_pass.n_out;
  const int per_sm = int(std::min<uint64_t>(uint64_t(MINB), (uint64_t(n_tiles) + num_sms - 1) / num_sms));
  const size_t smem_max = tile_smem_max<Real, KMAX>(MINB, per_sm);
  size_t smem = tile_smem_base<Real, KMAX>(MINB) +
                sizeof(uint32_t) * kStageTabWords * size_t(host_pass.stage_end - host_pass.stage_begin);
  if constexpr (WAY == 2) {
    if (!TileCopy<Real, KMAX>::fits(host_pass))
      return launch_tile_pass_cfg<Real, KMAX, MINB, 1>(amp, host_pass, d_prog, stream, num_sms);
  }
  if constexpr (WAY > 0) {
    smem = tile_smem_base<Real, KMAX>(MINB) + sizeof(ProgWord) * size_t(host_pass.prog_words);
    if (smem > smem_max) return launch_tile_pass_cfg<Real, KMAX, MINB, 0>(amp, host_pass, d_prog, stream, num_sms);
  }
  // the shared-memory limit is a per-device attribute: set once per device
  static PerDeviceOnce<cudaError_t> attr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = attr.get(dev, [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          int(tile_smem_max<Real, KMAX>(MINB, 1))); },
               cudaErrorInvalidDevice);
  if (e != cudaSuccess) return e;
  const unsigned grid = std::min<unsigned>(n_tiles, unsigned(num_sms) * MINB);
  uint64_t out_mask = 0, step = 0;  // qubits outside the tile; the grid size over them
  for (int j = 0; j < host_pass.n_out; ++j) {
    out_mask |= 1ull << host_pass.qout[j];
    step |= uint64_t((grid >> j) & 1u) << host_pass.qout[j];
  }
  // The pass may start while the kernel before it on the stream drains (its CTAs
  // load their tables, then wait for that kernel to complete).
  cudaLaunchAttribute pdl{};
  pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &pdl;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, amp, host_pass, reinterpret_cast<const uint4*>(d_prog), n_tiles,
                            out_mask, step);
}

template <typename Real>
static cudaError_t launch_tile_pass_t(Real* amp, const PassRec& host_pass, const ProgWord* d_prog,
                                      cudaStream_t stream, int num_sms) {
  constexpr int K = tile_kmax_full<Real>();
  constexpr DType dt = sizeof(Real) == 4 ? DType::C64 : DType::C128;
  constexpr int W = sizeof(Real) == 8 ? 2 : 1;
  switch (tile_launch_config(dt, tile_config_get(dt), host_pass.k, host_pass.n_out, num_sms)) {
    case 4: return launch_tile_pass_cfg<Real, K - 1, 4, W>(amp, host_pass, d_prog, stream, num_sms);
    case 2: return launch_tile_pass_cfg<Real, K, 2, W>(amp, host_pass, d_prog, stream, num_sms);
    default: return launch_tile_pass_cfg<Real, K, 1, 1>(amp, host_pass, d_prog, stream, num_sms);
  }
}

cudaError_t launch_tile_pass(DType dt, void* amp, const PassRec& host_pass, const ProgWord* d_prog,
                             cudaStream_t stream, int num_sms) {
  if (dt == DType::C64) return launch_tile_pass_t<float>(static_cast<float*>(amp), host_pass, d_prog, stream, num_sms);
  return launch_tile_pass_t<double>(static_cast<double*>(amp), host_pass, d_prog, stream, num_sms);
}

static int tile_kmax_for(DType dt) {
  const int full = dt == DType::C64 ? 13 : 12, set = tile_config_get(dt);
  return set == 4 || (set == 0 && dt == DType::C64) ? full - 1 : full;
}

// From this size on a complex64 pass is long enough (32 MB of state) for its HBM
// time to matter and for a second plan to be worth building.
constexpr int kWideTileMinQubits = 22;

// Complex64 tiles of 2^12 amplitudes are the better ones per pass (four CTAs of
// 128 threads against two of 256: 24-qubit brickwork 574 against 631 us on 4 passes
// either way), 2^13 save passes.  Taken when they save at least a fifth of the
// passes and stages too: 27-qubit phase estimation (7 passes and 19 stages instead
// of 10 and 22) 5.55 against 7.48 ms.  With the passes alone fewer they lose:
// 25-qubit Ising evolution of 10 steps (12 and 40 instead of 15 and 38) 3.30 against
// 3.17 ms, of 5 steps (6 and 21 instead of 8 and 20) 1.70 against 1.54.  A ratio of
// passes does not separate every case: phase estimation of 24 and 25 qubits (6
// passes for 7, 7 for 8) is refused and would take 0.65 for 0.85 ms and 1.36 for
// 1.81, that of 26 qubits would lose 6 %.
bool build_tile_plan_for(const std::vector<Op>& ops, int n, DType dt, TilePlan* out, std::string* err,
                         const std::function<bool(const TilePlan&)>& enough) {
  if (!build_tile_plan(ops, n, dt, tile_kmax_for(dt), out, err)) return false;
  if (dt != DType::C64 || tile_config_get(dt) != 0 || n < kWideTileMinQubits || out->passes.size() < 2) return true;
  if (enough && enough(*out)) return true;
  TilePlan wide;
  if (build_tile_plan(ops, n, dt, 13, &wide, err) && 5 * wide.passes.size() <= 4 * out->passes.size() &&
      wide.stats.stages < out->stats.stages)
    *out = std::move(wide);
  return true;
}

}  // namespace nqpu
