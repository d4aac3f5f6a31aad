// Test infrastructure: the engine's host code (engine.cpp) on a CUDA runtime of
// this file's own, without a GPU.  Device memory is host memory; work queued on a
// stream runs as late as the runtime allows, when the stream is waited for.  The
// kernels' launchers only record what the checks below ask about.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "engine.h"
#include "fused.h"
#include "tcrun.h"

using namespace nqpu;

namespace {
std::map<cudaStream_t, std::deque<std::function<void()>>> g_queue;
int g_fail_malloc = -1;   // the allocation that fails, counted from now on
int g_fail_measure = -1;  // the measurement launch that fails
int g_tile_cfg = 0;       // tile configuration; 1: plans on 11 bits here, else 12
int g_plans = 0;          // tiled plans built
int g_tc_runs = 0;        // circuits run in the tensor mode
uint64_t g_tc_passes = 0;  // of the tensor plan (0: the tensor mode does not take the circuit)
std::vector<uint32_t> g_words;  // program words of the tiled passes launched
void run(cudaStream_t st) {
  auto& q = g_queue[st];
  while (!q.empty()) {
    q.front()();
    q.pop_front();
  }
}
cudaStream_t new_stream() { return reinterpret_cast<cudaStream_t>(new int(0)); }
}  // namespace

// ---- CUDA runtime -----------------------------------------------------------
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_fail_malloc >= 0 && g_fail_malloc-- == 0) return cudaErrorMemoryAllocation;
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = new_stream(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { g_queue.erase(s); delete reinterpret_cast<int*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  for (auto& kv : g_queue) run(kv.first);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* h, size_t n, cudaMemcpyKind, cudaStream_t s) {
  g_queue[s].push_back([=] { std::memcpy(d, h, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* h, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, h, n, k, nullptr); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
  g_queue[s].push_back([=] { std::memset(d, v, n); });
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaErrorNotSupported; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaErrorNotSupported; }
}

// ---- launchers --------------------------------------------------------------
namespace nqpu {
double next_random_f64() { return 0.5; }
size_t reduce_scratch_bytes(int) { return 4096; }
int tile_config_get(DType) { return g_tile_cfg; }
bool build_tile_plan_for(const std::vector<Op>& ops, int n, DType dt, TilePlan* out, std::string* err,
                         const std::function<bool(const TilePlan&)>&) {
  ++g_plans;
  return build_tile_plan(ops, n, dt, g_tile_cfg == 1 ? 11 : 12, out, err);
}
cudaError_t launch_tile_pass(DType, void*, const PassRec& P, const ProgWord* prog, cudaStream_t, int) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(prog + P.prog_begin);
  g_words.insert(g_words.end(), w, w + 4 * P.prog_words);
  return cudaSuccess;
}
cudaError_t launch_pergate(DType, void*, int, const Op&, bool, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_set_basis(DType, void*, int, uint64_t, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_scale(DType, void*, int, double, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_collapse(DType, void*, int, int, int, double, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_measure_collapse(DType, void*, int, int, const double*, double, bool, double* result, cudaStream_t s,
                                    int) {
  if (g_fail_measure >= 0 && g_fail_measure-- == 0) return cudaErrorLaunchOutOfResources;
  if (result) g_queue[s].push_back([=] { result[0] = 1.0; });
  return cudaSuccess;
}
cudaError_t launch_probabilities(DType, const void*, uint64_t, double*, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_convert(DType, const void*, DType, void*, uint64_t, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_zsums(DType, const void*, int, double*, double*, cudaStream_t, int) { return cudaSuccess; }
cudaError_t launch_inner(DType, const void*, DType, const void*, int, double*, double*, cudaStream_t, int) {
  return cudaSuccess;
}
cudaError_t launch_pauli(DType, const void*, int, uint64_t, uint64_t, uint64_t, double*, double*, cudaStream_t, int) {
  return cudaSuccess;
}
void pauli_plan(DType, const PauliString*, size_t, int, PauliPlan*, std::vector<PauliString>*) {}
cudaError_t launch_pauli_sum(DType, const void*, int, const PauliSet*, const PauliPlan&, const PauliTerm*, double*, double*,
                             cudaStream_t, int) {
  return cudaSuccess;
}
cudaError_t launch_sample(DType, const void*, int, const double*, uint32_t, double*, uint64_t*, cudaStream_t, int) {
  return cudaSuccess;
}
bool fused_plan_build(const std::vector<Op>&, int, DType, cudaStream_t, void**, PlanStats*) { return false; }
bool fused_plan_stats(const std::vector<Op>&, int, DType, PlanStats*) { return false; }
void fused_plan_free(void*) {}
cudaError_t fused_run(void*, StateImpl*, std::vector<cudaEvent_t>*) { return cudaSuccess; }
bool tc_plan_build(const std::vector<Op>&, int, DType, cudaStream_t, void** plan, PlanStats*) {
  *plan = nullptr;
  return true;
}
bool tc_plan_stats(const std::vector<Op>&, int, DType, PlanStats* st) {
  st->passes = st->stages = g_tc_passes;
  return g_tc_passes > 0;
}
void tc_plan_free(void*) {}
cudaError_t tc_run(void*, StateImpl*, std::vector<cudaEvent_t>*) {
  ++g_tc_runs;
  return cudaSuccess;
}
}  // namespace nqpu

// ---- checks (0: as it should be) ---------------------------------------------
// A plan table is in device memory when its upload returns, whatever its size.
extern "C" int check_upload(int bytes) {
  std::vector<unsigned char> h(size_t(bytes) + 1, 0xA5);
  cudaStream_t st = new_stream();
  void* d = nullptr;
  if (upload_table(&d, h.data(), size_t(bytes), st) != cudaSuccess || !d) return 1;
  if (std::memcmp(d, h.data(), size_t(bytes)) != 0) return 2;
  for (auto& kv : g_queue)
    if (!kv.second.empty()) return 3;
  cudaFree(d);
  cudaStreamDestroy(st);
  return 0;
}

static bool idle(StateImpl* s) { return g_queue[s->stream].empty(); }

// H, measurement, H, measurement, H: the third segment's plan upload fails (what
// = 0) or the second measurement's launch (1); then one of a whole register's
// measurements (2).  Nothing may stay queued that writes to the state's buffers, and
// the first error is what the call returns.
extern "C" int check_measure_error(int what) {
  StateImpl* s = state_new(6, DType::C64);
  CircuitImpl c;
  c.n = 6;
  for (int i = 0; i < 5; ++i) {
    GateRec g;
    g.code = i % 2 ? G_MEASURE : G_H;
    c.gates.push_back(g);
  }
  std::vector<uint32_t> out(6);
  g_fail_malloc = what == 0 ? 2 : -1;
  g_fail_measure = what == 1 ? 1 : what == 2 ? 3 : -1;
  const cudaError_t e = what == 2 ? state_measure_all(s, out.data())
                                  : circuit_run(&c, s, NQPU_MODE_TILED, nullptr, &out);
  g_fail_malloc = g_fail_measure = -1;
  if (e != (what == 0 ? cudaErrorMemoryAllocation : cudaErrorLaunchOutOfResources)) return 1;
  if (!idle(s)) return 2;
  // without a failure the same circuit's outcomes all arrive
  out.clear();
  if (circuit_run(&c, s, NQPU_MODE_TILED, nullptr, &out) != cudaSuccess || out.size() != 2) return 3;
  if (out[0] != 1 || out[1] != 1) return 4;
  state_free(s);
  return 0;
}

// Six layers of U3s and CNOTs in a ring.
static std::vector<GateRec> layers(int n) {
  std::vector<GateRec> gates;
  for (int l = 0; l < 6; ++l)
    for (int q = 0; q < n; ++q) {
      GateRec g;
      g.code = G_U3;
      g.q[0] = q;
      g.p[0] = 0.3 + q + l, g.p[1] = 0.7 * q - l, g.p[2] = 1.1 + l * q;
      gates.push_back(g);
      g.code = G_CX;
      g.nq = 2;
      g.q[1] = (q + 1) % n;
      gates.push_back(g);
    }
  return gates;
}

// AUTO builds one tiled plan for a circuit that it runs in the tiled mode, none for
// its second run, and the programs are the tiled mode's own.
extern "C" int check_auto_plans_once(int n) {
  StateImpl* s = state_new(uint32_t(n), DType::C64);
  const std::vector<GateRec> gates = layers(n);
  CircuitImpl a, b;
  a.n = b.n = uint32_t(n);
  a.gates = b.gates = gates;
  g_tc_passes = 1000;
  g_plans = 0;
  g_words.clear();
  if (circuit_run(&a, s, NQPU_MODE_AUTO) != cudaSuccess || g_plans != 1 || g_words.empty()) return 1;
  const std::vector<uint32_t> words = std::move(g_words);
  g_words.clear();
  if (circuit_run(&a, s, NQPU_MODE_AUTO) != cudaSuccess || g_plans != 1 || g_words != words) return 2;
  g_words.clear();
  if (circuit_run(&b, s, NQPU_MODE_TILED) != cudaSuccess || g_plans != 2 || g_words != words) return 3;
  g_tc_passes = 0;
  state_free(s);
  return 0;
}

// AUTO chooses again when the tile configuration that the choice was made for has
// changed, and keeps its choice while it has not: a tensor plan priced between the
// tiled plans of two tile sizes.
extern "C" int check_auto_follows_tiles() {
  const int n = 22;
  StateImpl* s = state_new(n, DType::C64);
  CircuitImpl c;
  c.n = n;
  c.gates = layers(n);
  const std::vector<Op> ops = lower_circuit(c.gates);
  auto mode_at = [&](int cfg) {
    g_tile_cfg = cfg;
    return auto_mode_for(ops, n, DType::C64);
  };
  g_tc_passes = 0;
  do ++g_tc_passes;
  while (g_tc_passes < 1000 && mode_at(0) == NQPU_MODE_TENSOR);  // dearer than the 12-bit plan,
  if (mode_at(0) != NQPU_MODE_TILED || mode_at(1) != NQPU_MODE_TENSOR) return 1;  // cheaper than the 11-bit one
  auto tensor_runs = [&](int cfg) {
    g_tile_cfg = cfg;
    g_tc_runs = 0;
    return circuit_run(&c, s, NQPU_MODE_AUTO) == cudaSuccess ? g_tc_runs : -1;
  };
  int rc = 0;
  if (tensor_runs(0) != 0) rc = 2;
  else if (tensor_runs(1) != 1) rc = 3;
  else if (tensor_runs(0) != 0) rc = 4;
  g_plans = 0;
  if (!rc && (tensor_runs(0) != 0 || g_plans != 0)) rc = 5;
  g_tile_cfg = 0;
  g_tc_passes = 0;
  state_free(s);
  return rc;
}

// The configuration a pass is launched in holds its tiles whatever is set, and is the
// set one wherever that holds them.
extern "C" int check_launch_config() {
  for (DType dt : {DType::C64, DType::C128}) {
    const int full = dt == DType::C64 ? 13 : 12;
    for (int set : {0, 1, 2, 4})
      for (int k = 5; k <= full; ++k)
        for (int n_out : {0, 3, 7, 8, 20}) {
          const int cfg = tile_launch_config(dt, set, k, n_out, 148);
          if (cfg != 1 && cfg != 2 && cfg != 4) return 1;
          if (k > (cfg == 4 ? full - 1 : full)) return 2;
          if (set != 0 && cfg != set && !(set == 4 && k == full)) return 3;
        }
  }
  return 0;
}

// Per-gate launches alternate their direction from 128 MB of state on, and not below.
extern "C" int check_sweeps() {
  StateImpl s;
  for (size_t mb : {1, 64, 127}) {
    s.bytes = mb << 20;
    for (int i = 0; i < 4; ++i)
      if (s.next_sweep()) return 1;
  }
  for (size_t mb : {128, 4096}) {
    s.bytes = mb << 20;
    bool last = s.sweep;
    for (int i = 0; i < 4; ++i) {
      const bool now = s.next_sweep();
      if (now == last) return 2;
      last = now;
    }
  }
  return 0;
}
