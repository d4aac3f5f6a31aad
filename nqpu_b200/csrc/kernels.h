// Launch wrappers of the sm_100a kernels, called by the host engine.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <functional>
#include <vector>
#include "planner.h"
#include "sv_types.h"

namespace nqpu {

// Arguments of a per-gate launch (passed by value).
struct PGArgs {
  uint64_t n_items;   // work items (index sets) of the launch
  uint64_t setmask;   // bits forced to one (controls)
  union {
    uint64_t cmask;   // controls checked per amplitude (elementwise kernels)
    uint64_t flip;    // X: n_items - 1 in a launch that runs from the far end, else 0
  };
  int32_t npos;       // zero-bit insert positions, ascending
  int32_t pos[8];
  int32_t t0, t1;
  double m[32];
};

// --- per-gate path -----------------------------------------------------------
// State size from which successive launches sweep in alternate directions.
constexpr size_t kSweepBytes = size_t(128) << 20;
// `rev`: sweep the state from its far end (callers alternate from gate to gate).
cudaError_t launch_pergate(DType dt, void* amp, int n, const Op& op, bool rev, cudaStream_t s, int num_sms);

// --- tiled pass path ---------------------------------------------------------
// CTA configuration of the tiled pass kernel (1: one CTA per SM, double-buffered
// tiles; 2: two CTAs per SM, single-buffered; 4: four on half-size tiles; 0, the
// default: chosen per plan and launch).
void tile_config_set(DType dt, int minb);
int tile_config_get(DType dt);
// The configuration (1, 2 or 4) that a pass of 2^k-amplitude tiles over 2^n_out of
// them runs in where `set` is set.  One that was planned on larger tiles than 4
// takes runs in 2: the setting may change after a plan was made, under a request
// that waits for its launch or in another thread.
inline int tile_launch_config(DType dt, int set, int k, int n_out, int num_sms) {
  const int full = dt == DType::C64 ? 13 : 12;
  if (set == 0 && dt == DType::C128) return (uint64_t(1) << n_out) <= uint64_t(num_sms) ? 1 : 2;
  if (set == 0 || set == 4) return k == full ? 2 : 4;
  return set;
}
// Tiled plan of the tile size in force for the dtype.
// (`enough`: asked with the first plan, true spares the search for a better one)
bool build_tile_plan_for(const std::vector<Op>& ops, int n, DType dt, TilePlan* out, std::string* err,
                         const std::function<bool(const TilePlan&)>& enough = nullptr);
// One pass; d_prog is the plan's program table in device memory.
cudaError_t launch_tile_pass(DType dt, void* amp, const PassRec& host_pass, const ProgWord* d_prog,
                             cudaStream_t stream, int num_sms);

// --- state utilities ---------------------------------------------------------
cudaError_t launch_set_basis(DType dt, void* amp, int n, uint64_t index, cudaStream_t s, int num_sms);
cudaError_t launch_scale(DType dt, void* amp, int n, double factor, cudaStream_t s, int num_sms);
// zero amplitudes whose bit q differs from `keep`, scale the rest by `factor`
cudaError_t launch_collapse(DType dt, void* amp, int n, int q, int keep, double factor,
                            cudaStream_t s, int num_sms);
// Measure qubit q with the uniform draw r from launch_zsums' sums (device memory):
// collapse, and with `flip` move outcome 1 to |0>.  result[0..1] (device or pinned
// host memory, may be null) = outcome, its probability.
cudaError_t launch_measure_collapse(DType dt, void* amp, int n, int q, const double* sums, double r, bool flip,
                                    double* result, cudaStream_t s, int num_sms);
// |a_i|^2 for `count` amplitudes starting at `amp` (already offset by the caller).
cudaError_t launch_probabilities(DType dt, const void* amp, uint64_t count, double* out,
                                 cudaStream_t s, int num_sms);
// Convert `count` amplitudes between dtypes (either may equal the other).
cudaError_t launch_convert(DType src_dt, const void* src, DType dst_dt, void* dst, uint64_t count,
                           cudaStream_t s, int num_sms);

// --- FP64 reductions ---------------------------------------------------------
// All-<Z_i>: a warp works on chunks of kZsChunkVecs 128-bit vectors; the scratch
// holds one row per value (n + 1 of them) of at most kZsMaxBlocks block partials.
constexpr uint64_t kZsChunkVecs = 32 * 8;  // lanes x vectors per lane
constexpr int kZsMaxBlocks = 1024;
// Doubles of all-<Z_i> scratch for an n-qubit state.
constexpr size_t zsums_scratch_doubles(int n) { return size_t(kZsMaxBlocks) * size_t(n + 1); }
// Scratch bytes every reduction below needs on an n-qubit state.
size_t reduce_scratch_bytes(int n);
// out[v] = sum over b < nblk of part[v * nblk + b] (one block, fixed order).
cudaError_t launch_sum_rows(const double* part, int nvals, int nblk, double* out, cudaStream_t s);
// out[0] = sum |a|^2, out[1+q] = sum over amplitudes with bit q set of |a|^2, q < n.
// `out` here and in launch_inner is device memory or pinned host memory.
cudaError_t launch_zsums(DType dt, const void* amp, int n, double* scratch, double* out,
                         cudaStream_t s, int num_sms);
// out[0..1] = sum conj(a) b (re, im)
cudaError_t launch_inner(DType dta, const void* a, DType dtb, const void* b, int n,
                         double* scratch, double* out, cudaStream_t s, int num_sms);
// Pauli-string expectation (R/lib.rs:465 semantics): xmask = X|Y positions,
// zmask = Z|Y positions, ymask = Y positions.  out[0] = real part.
cudaError_t launch_pauli(DType dt, const void* amp, int n, uint64_t xmask, uint64_t zmask,
                         uint64_t ymask, double* scratch, double* out, cudaStream_t s,
                         int num_sms);

// --- Pauli sums (kernels_pauli.cu) -------------------------------------------
struct PauliString {
  uint64_t x, z, y;  // X|Y positions, Z|Y positions, Y positions
  double c;
};
// A register set of the Pauli-sum kernel: a thread holds the 16 amplitudes that
// differ in the four index bits rbit (ascending) and evaluates on them every
// term whose X|Y positions lie in those bits.  Terms [beg[m], beg[m + 1]) have
// X|Y positions m (a mask over rbit); beg[0]..beg[1] are diagonal terms, sorted
// by their Z positions within rbit, dbeg[k] the first with positions >= k.
struct PauliSet {
  uint16_t beg[17];
  uint16_t dbeg[17];
  uint16_t xused, dused;  // bit m: the list of X|Y (diagonal: Z) positions m is not empty
  uint16_t plain;         // bit b: a single X on bit b alone, its coefficient in cx[b] (not in the lists)
  alignas(4) uint8_t rbit[4];
  double cx[4];
};
// One term: z = Z|Y positions outside the set's bits | those inside << 60 |
// (odd number of Y's) << 59; c = coefficient with the pair factor and the sign
// of i^ny folded in.
struct PauliTerm {
  uint64_t z;
  double c;
};
constexpr int kPauliMaxTerms = 65535;  // of one launch (16-bit offsets)
struct PauliPlan {
  std::vector<PauliSet> sets;
  std::vector<PauliTerm> terms;
};
// Split a Pauli sum on n >= 4 qubits into register sets; terms that run better by
// themselves (X|Y positions on more than four qubits, or on the lowest ones of a
// large complex128 state and alone there) are left in `wide` (at most
// kPauliMaxTerms strings per call).
void pauli_plan(DType dt, const PauliString* strings, size_t count, int n, PauliPlan* plan,
                std::vector<PauliString>* wide);
// out[0] = the plan's sum over the state; d_sets / d_terms are the plan's tables
// in device memory.
cudaError_t launch_pauli_sum(DType dt, const void* amp, int n, const PauliSet* d_sets, const PauliPlan& plan,
                             const PauliTerm* d_terms, double* scratch, double* out, cudaStream_t s, int num_sms);

// Sampling with given uniforms: out[s] = first i with u[s] < cumsum_i, else 2^n-1.
cudaError_t launch_sample(DType dt, const void* amp, int n, const double* d_uniforms,
                          uint32_t shots, double* scratch, uint64_t* d_out, cudaStream_t s,
                          int num_sms);

}  // namespace nqpu
