// Engine objects: device context, state allocation, reductions glue and the
// circuit runner (tiled passes / per-gate / fused).
#include "engine.h"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include "device_once.h"
#include "fused.h"
#include "kernels.h"
#include "tcpass.h"
#include "tcrun.h"
#include "tileprog.h"

namespace nqpu {

namespace {
std::once_flag g_dev_once;
bool g_dev_ok = false;

void dev_init() {
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0) {
    cudaGetLastError();
    g_dev_ok = false;
    return;
  }
  g_dev_ok = true;
}
}  // namespace

bool device_ready() {
  std::call_once(g_dev_once, dev_init);
  return g_dev_ok;
}

// SM count of the current device (grids are sized in multiples of it), read
// once per device.
int device_sms() {
  static PerDeviceOnce<int> sms;
  int dev = 0;
  if (!device_ready() || cudaGetDevice(&dev) != cudaSuccess) return 148;
  return sms.get(dev, [dev] {
    int v = 0;
    return (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0) ? v : 148;
  }, 148);
}

cudaError_t upload_table(void** dev, const void* host, size_t bytes, cudaStream_t st) {
  cudaError_t e = cudaMalloc(dev, std::max<size_t>(16, bytes));
  if (e != cudaSuccess || bytes == 0) return e;
  e = cudaMemcpyAsync(*dev, host, bytes, cudaMemcpyHostToDevice, st);
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

StateImpl* state_new(uint32_t n, DType dt) {
  if (!device_ready()) return nullptr;
  auto* s = new (std::nothrow) StateImpl();
  if (!s) return nullptr;
  s->n = n;
  s->dt = dt;
  s->bytes = size_t(amp_bytes(dt)) << n;
  bool ok = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) == cudaSuccess;
  ok = ok && cudaMalloc(&s->amp, s->bytes) == cudaSuccess;
  ok = ok && cudaMalloc(reinterpret_cast<void**>(&s->scratch), reduce_scratch_bytes(int(n))) == cudaSuccess;
  ok = ok && cudaMalloc(reinterpret_cast<void**>(&s->d_small), kSmallDoubles * sizeof(double)) == cudaSuccess;
  ok = ok && cudaMallocHost(reinterpret_cast<void**>(&s->h_small), kSmallDoubles * sizeof(double)) == cudaSuccess;
  ok = ok && launch_set_basis(dt, s->amp, int(n), 0, s->stream, device_sms()) == cudaSuccess;
  ok = ok && cudaStreamSynchronize(s->stream) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    state_free(s);
    return nullptr;
  }
  return s;
}

void state_free(StateImpl* s) {
  if (!s) return;
  if (s->stream) cudaStreamSynchronize(s->stream);
  if (s->amp) cudaFree(s->amp);
  if (s->scratch) cudaFree(s->scratch);
  if (s->d_small) cudaFree(s->d_small);
  if (s->h_small) cudaFreeHost(s->h_small);
  if (s->d_tab) cudaFree(s->d_tab);
  if (s->d_uni) cudaFree(s->d_uni);
  if (s->d_shots) cudaFree(s->d_shots);
  if (s->run_norm) cudaFree(s->run_norm);
  if (s->run_err) cudaFree(s->run_err);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

cudaError_t state_run_scratch(StateImpl* s, size_t doubles, double** norm, int** err) {
  cudaError_t e;
  if (s->run_norm_cap < doubles) {
    // the old buffer may back a run still queued on the state's stream
    if (s->run_norm && (e = cudaStreamSynchronize(s->stream)) != cudaSuccess) return e;
    if (s->run_norm) cudaFree(s->run_norm);
    s->run_norm = nullptr;
    s->run_norm_cap = 0;
    if ((e = cudaMalloc(reinterpret_cast<void**>(&s->run_norm), doubles * sizeof(double))) != cudaSuccess) return e;
    s->run_norm_cap = doubles;
  }
  if (!s->run_err && (e = cudaMalloc(reinterpret_cast<void**>(&s->run_err), sizeof(int))) != cudaSuccess) return e;
  // the expiry flag of an earlier run is cleared, so this run reports its own
  if ((e = cudaMemsetAsync(s->run_err, 0, sizeof(int), s->stream)) != cudaSuccess) return e;
  *norm = s->run_norm;
  *err = s->run_err;
  return cudaSuccess;
}

cudaError_t state_run_error(StateImpl* s) {
  if (!s->run_err) return cudaSuccess;
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, s->run_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return e;
  return h ? cudaErrorLaunchTimeout : cudaSuccess;
}

cudaError_t state_zsums(const StateImpl* s, double* zs, double* total) {
  const int n = int(s->n);
  cudaError_t e = launch_zsums(s->dt, s->amp, n, s->scratch, s->h_small, s->stream, device_sms());
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return e;
  if (zs) std::memcpy(zs, s->h_small, sizeof(double) * (n + 1));
  if (total) *total = s->h_small[0];
  return cudaSuccess;
}

cudaError_t state_queue_measure(StateImpl* s, uint32_t qubit, bool flip, double* result) {
  const double r = next_random_f64();
  cudaError_t e = launch_zsums(s->dt, s->amp, int(s->n), s->scratch, s->d_small, s->stream, device_sms());
  if (e != cudaSuccess) return e;
  return launch_measure_collapse(s->dt, s->amp, int(s->n), int(qubit), s->d_small, r, flip, result, s->stream,
                                 device_sms());
}

cudaError_t state_measure(StateImpl* s, uint32_t qubit, uint32_t* outcome, double* probability) {
  double* res = s->h_small + kSmallTable;
  cudaError_t e = state_queue_measure(s, qubit, false, res);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return e;
  *outcome = uint32_t(res[0]);
  if (probability) *probability = res[1];
  return cudaSuccess;
}

cudaError_t state_measure_all(StateImpl* s, uint32_t* outcomes) {
  double* res = s->h_small + kSmallTable;
  static_assert(kSmallTable + 2 * size_t(kMaxQubits) <= kSmallDoubles, "room for every qubit's result");
  for (uint32_t q = 0; q < s->n; ++q) {
    const cudaError_t e = state_queue_measure(s, q, false, res + 2 * q);
    if (e != cudaSuccess) {
      cudaStreamSynchronize(s->stream);  // the queued ones write to the staging buffer
      return e;
    }
  }
  const cudaError_t e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return e;
  for (uint32_t q = 0; q < s->n; ++q) outcomes[q] = uint32_t(res[2 * q]);
  return cudaSuccess;
}

cudaError_t state_reset_qubit(StateImpl* s, uint32_t qubit) {
  std::vector<double> z(s->n + 1);
  cudaError_t e = state_zsums(s, z.data(), nullptr);
  if (e != cudaSuccess) return e;
  const double keep = z[0] - z[1 + qubit];  // norm of the |0> half
  const double f = keep > 0.0 ? 1.0 / std::sqrt(keep) : 1.0;
  return launch_collapse(s->dt, s->amp, int(s->n), int(qubit), 0, f, s->stream, device_sms());
}

// One string that no register set holds (or a state of fewer than four qubits).
static cudaError_t pauli_direct(const StateImpl* s, const PauliString& p, double* out) {
  cudaError_t e = launch_pauli(s->dt, s->amp, int(s->n), p.x, p.z, p.y, s->scratch, s->h_small, s->stream, device_sms());
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e == cudaSuccess) *out += p.c * s->h_small[0];
  return e;
}

static cudaError_t pauli_sum(StateImpl* s, const std::vector<PauliString>& strings, double* out);

// The kernel adds coefficients up before they meet the amplitudes and doubles those
// of pairs: near the ends of the type's range it works on coefficients scaled by a
// power of two, so that a sum overflows or vanishes only where its value does.
cudaError_t state_pauli_sum(StateImpl* s, const std::vector<PauliString>& strings, double* out) {
  double most = 0.0;
  for (const PauliString& p : strings) most = std::max(most, std::fabs(p.c));
  constexpr int kRoom = 900;  // of 1023: 2^123 for the sum of 2^32 terms and for the doubling
  const int e = most > 0.0 ? std::ilogb(most) : 0;
  const int shift = e > kRoom ? e - kRoom : e < -kRoom ? e + kRoom : 0;
  if (shift == 0) return pauli_sum(s, strings, out);
  std::vector<PauliString> scaled = strings;
  for (PauliString& p : scaled) p.c = std::ldexp(p.c, -shift);
  const cudaError_t r = pauli_sum(s, scaled, out);
  *out = std::ldexp(*out, shift);
  return r;
}

static cudaError_t pauli_sum(StateImpl* s, const std::vector<PauliString>& strings, double* out) {
  *out = 0.0;
  cudaError_t e;
  if (s->n < 4) {
    for (const PauliString& p : strings)
      if ((e = pauli_direct(s, p, out)) != cudaSuccess) return e;
    return cudaSuccess;
  }
  PauliPlan plan;
  std::vector<PauliString> wide;
  for (size_t lo = 0; lo < strings.size(); lo += kPauliMaxTerms) {
    pauli_plan(s->dt, strings.data() + lo, std::min<size_t>(kPauliMaxTerms, strings.size() - lo), int(s->n), &plan, &wide);
    for (const PauliString& p : wide)
      if ((e = pauli_direct(s, p, out)) != cudaSuccess) return e;
    if (plan.sets.empty()) continue;
    // tables: terms (16 bytes each), then the sets
    const size_t tb = plan.terms.size() * sizeof(PauliTerm), bytes = tb + plan.sets.size() * sizeof(PauliSet);
    char* dev = reinterpret_cast<char*>(s->d_small + kSmallTable);
    std::vector<char> big;
    char* host = reinterpret_cast<char*>(s->h_small + kSmallTable);
    if (bytes > (kSmallDoubles - kSmallTable) * sizeof(double)) {
      if (s->tab_cap < bytes) {
        if (s->d_tab) cudaFree(s->d_tab);  // earlier sums have returned, so nothing queued reads it
        s->d_tab = nullptr;
        s->tab_cap = 0;
        if ((e = cudaMalloc(&s->d_tab, bytes)) != cudaSuccess) return e;
        s->tab_cap = bytes;
      }
      dev = static_cast<char*>(s->d_tab);
      big.resize(bytes);
      host = big.data();
    }
    std::memcpy(host, plan.terms.data(), tb);
    std::memcpy(host + tb, plan.sets.data(), bytes - tb);
    if ((e = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s->stream)) != cudaSuccess) return e;
    e = launch_pauli_sum(s->dt, s->amp, int(s->n), reinterpret_cast<const PauliSet*>(dev + tb), plan,
                         reinterpret_cast<const PauliTerm*>(dev), s->scratch, s->h_small, s->stream, device_sms());
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return e;
    *out += s->h_small[0];
  }
  return cudaSuccess;
}

cudaError_t state_inner(const StateImpl* a, const StateImpl* b, double* out2) {
  cudaError_t e = cudaStreamSynchronize(b->stream);
  if (e != cudaSuccess) return e;
  e = launch_inner(a->dt, a->amp, b->dt, b->amp, int(a->n), a->scratch, a->h_small, a->stream, device_sms());
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(a->stream);
  if (e != cudaSuccess) return e;
  out2[0] = a->h_small[0];
  out2[1] = a->h_small[1];
  return cudaSuccess;
}

cudaError_t state_sample(const StateImpl* sc, const double* uniforms, uint32_t shots, uint64_t* out) {
  StateImpl* s = const_cast<StateImpl*>(sc);
  cudaError_t e;
  if (2 * size_t(shots) <= kSmallDoubles - kSmallTable) {
    // uniforms staged in pinned memory, outcomes written there by the kernel: a
    // copy from or to pageable memory costs about 10 us each way
    double* hu = s->h_small + kSmallTable;
    double* du = s->d_small + kSmallTable;
    uint64_t* ho = reinterpret_cast<uint64_t*>(hu + shots);
    std::memcpy(hu, uniforms, sizeof(double) * shots);
    if ((e = cudaMemcpyAsync(du, hu, sizeof(double) * shots, cudaMemcpyHostToDevice, s->stream)) != cudaSuccess) return e;
    if ((e = launch_sample(s->dt, s->amp, int(s->n), du, shots, s->scratch, ho, s->stream, device_sms())) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s->stream)) != cudaSuccess) return e;
    std::memcpy(out, ho, sizeof(uint64_t) * shots);
    return cudaSuccess;
  }
  if (s->shot_cap < shots) {
    e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return e;
    if (s->d_uni) cudaFree(s->d_uni);
    if (s->d_shots) cudaFree(s->d_shots);
    s->d_uni = nullptr;
    s->d_shots = nullptr;
    s->shot_cap = 0;
    if ((e = cudaMalloc(reinterpret_cast<void**>(&s->d_uni), sizeof(double) * shots)) != cudaSuccess) return e;
    if ((e = cudaMalloc(reinterpret_cast<void**>(&s->d_shots), sizeof(uint64_t) * shots)) != cudaSuccess) return e;
    s->shot_cap = shots;
  }
  if ((e = cudaMemcpyAsync(s->d_uni, uniforms, sizeof(double) * shots, cudaMemcpyHostToDevice, s->stream)) != cudaSuccess) return e;
  if ((e = launch_sample(s->dt, s->amp, int(s->n), s->d_uni, shots, s->scratch, s->d_shots, s->stream, device_sms())) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(out, s->d_shots, sizeof(uint64_t) * shots, cudaMemcpyDeviceToHost, s->stream)) != cudaSuccess) return e;
  return cudaStreamSynchronize(s->stream);
}

// Probabilities in chunks through a device buffer (the full 2^n FP64 vector may
// not fit next to the state).
cudaError_t state_probabilities(const StateImpl* s, double* out) {
  const uint64_t dim = 1ull << s->n;
  const uint64_t chunk = std::min<uint64_t>(dim, 1ull << 24);
  double* d = nullptr;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d), chunk * sizeof(double));
  if (e != cudaSuccess) return e;
  const size_t ab = amp_bytes(s->dt);
  for (uint64_t off = 0; off < dim && e == cudaSuccess; off += chunk) {
    const uint64_t cnt = std::min(chunk, dim - off);
    e = launch_probabilities(s->dt, static_cast<const char*>(s->amp) + off * ab, cnt, d, s->stream, device_sms());
    if (e == cudaSuccess) e = cudaMemcpyAsync(out + off, d, cnt * sizeof(double), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  }
  cudaFree(d);
  return e;
}

cudaError_t state_download_c128(const StateImpl* s, NqpuComplex* out) {
  const uint64_t dim = 1ull << s->n;
  if (dim * 16 <= (kSmallDoubles - kSmallTable) * sizeof(double)) {
    // a small register through the pinned buffer (no allocation, and a copy to
    // pageable memory costs several microseconds more)
    double* h = s->h_small + kSmallTable;
    cudaError_t e = s->dt == DType::C128
                        ? cudaMemcpyAsync(h, s->amp, dim * 16, cudaMemcpyDeviceToHost, s->stream)
                        : launch_convert(DType::C64, s->amp, DType::C128, h, dim, s->stream, device_sms());
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e == cudaSuccess) std::memcpy(static_cast<void*>(out), h, dim * 16);
    return e;
  }
  if (s->dt == DType::C128) {
    cudaError_t e = cudaMemcpyAsync(out, s->amp, dim * 16, cudaMemcpyDeviceToHost, s->stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s->stream);
  }
  const uint64_t chunk = std::min<uint64_t>(dim, 1ull << 22);
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, chunk * 16);
  if (e != cudaSuccess) return e;
  for (uint64_t off = 0; off < dim && e == cudaSuccess; off += chunk) {
    const uint64_t cnt = std::min(chunk, dim - off);
    e = launch_convert(DType::C64, static_cast<const char*>(s->amp) + off * 8, DType::C128, d, cnt, s->stream, device_sms());
    if (e == cudaSuccess) e = cudaMemcpyAsync(out + off, d, cnt * 16, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  }
  cudaFree(d);
  return e;
}

cudaError_t state_upload_c128(StateImpl* s, const NqpuComplex* in) {
  const uint64_t dim = 1ull << s->n;
  if (s->dt == DType::C128) {
    cudaError_t e = cudaMemcpyAsync(s->amp, in, dim * 16, cudaMemcpyHostToDevice, s->stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s->stream);
  }
  const uint64_t chunk = std::min<uint64_t>(dim, 1ull << 22);
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, chunk * 16);
  if (e != cudaSuccess) return e;
  for (uint64_t off = 0; off < dim && e == cudaSuccess; off += chunk) {
    const uint64_t cnt = std::min(chunk, dim - off);
    e = cudaMemcpyAsync(d, in + off, cnt * 16, cudaMemcpyHostToDevice, s->stream);
    if (e == cudaSuccess) e = launch_convert(DType::C128, d, DType::C64, static_cast<char*>(s->amp) + off * 8, cnt, s->stream, device_sms());
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  }
  cudaFree(d);
  return e;
}

// ---------------------------------------------------------------------------
// Circuits
// ---------------------------------------------------------------------------
static void plan_free(DevicePlan* p) {
  if (!p) return;
  if (p->d_prog) cudaFree(p->d_prog);
  if (p->fused) fused_plan_free(p->fused);
  if (p->tc) tc_plan_free(p->tc);
  delete p;
}

void circuit_free(CircuitImpl* c) {
  if (!c) return;
  cudaDeviceSynchronize();
  for (auto& kv : c->plans) plan_free(kv.second);
  delete c;
}

bool circuit_has_mid(const std::vector<GateRec>& gates) {
  for (const GateRec& g : gates)
    if (gate_is_mid(g.code)) return true;
  return false;
}

std::vector<Segment> circuit_segments(const std::vector<GateRec>& gates) {
  std::vector<Segment> segs;
  size_t b = 0;
  for (size_t i = 0; i < gates.size(); ++i)
    if (gate_is_mid(gates[i].code)) {
      segs.push_back(Segment{b, i, long(i)});
      b = i + 1;
    }
  segs.push_back(Segment{b, gates.size(), -1});
  return segs;
}

// The segment's plan; the tables of the fused and tensor modes are uploaded on `st`
// (those of the tiled mode by the caller; without a stream no mode uploads).  A
// tiled plan made for the same ops may be in p->tile already (auto_mode_for).
static bool plan_host(const CircuitImpl* c, const Segment& seg, uint32_t n, DType dt, int mode, cudaStream_t st,
                      DevicePlan* p) {
  p->ops = lower_circuit(std::vector<GateRec>(c->gates.begin() + long(seg.begin), c->gates.begin() + long(seg.end)));
  p->stats = PlanStats{};
  if (mode == NQPU_MODE_TILED && int(n) >= tile_min_qubits(dt)) {
    std::string err;
    p->ops = carry_phases(std::move(p->ops));
    p->tile_cfg = tile_config_get(dt);
    if (p->tile.passes.empty() && !build_tile_plan_for(p->ops, int(n), dt, &p->tile, &err)) return false;
    build_tile_prog(p->ops, &p->tile);
    p->stats = p->tile.stats;
  } else if (mode == NQPU_MODE_FUSED) {
    p->stats.ops = p->ops.size();
    return fused_plan_build(p->ops, int(n), dt, st, &p->fused, &p->stats);
  } else if (mode == NQPU_MODE_TENSOR) {
    return tc_plan_build(p->ops, int(n), dt, st, &p->tc, &p->stats);
  } else {
    p->stats.passes = p->ops.size();
    p->stats.ops = p->ops.size();
  }
  return true;
}

// NQPU_MODE_AUTO: the engine mode with the lower modelled device time (the
// counterpart of the reference's runtime-estimate backend choice,
// select_backend_estimated, backends/runtime/auto_simulator.rs:1452, among
// its statevector variants).  Both models are device time as U x work + launch
// cost, U = one HBM pass over the state (2 S bytes at 6.5 TB/s):
//   tiled   U (0.80 passes + 0.069 stages + 0.071 one-qubit 2x2s + 0.011
//           diagonal ops) + 11.2 us per pass + 1.1 us per stage
//   tensor  U (1.013 passes + 0.139 unitaries) + 16.8 us per pass + 34 us
// fitted (least squares of the relative error) to 42 measured complex64 circuits:
// brickwork, ansatz, Ising evolution and phase estimation of 14 to 28 qubits and
// two depths, none held out, with the kernels of that time (later ones took a few
// per cent off either side).  The fit is within 15 % for most, and picks the faster
// mode for every one of them: the tensor passes win on brickworks from 23 qubits on
// (26 qubits, 12 layers: 4.5 against 6.9 ms), the tiled ones everywhere else
// (30-qubit Ising evolution, 10 steps: 121 against 140 ms).  4x4 matrices and 2x2s
// with controls run as single records, priced at the 0.30 and 0.15 they
// measured as such.
int auto_mode_for(const std::vector<Op>& ops, uint32_t n, DType dt, TilePlan* plan) {
  if (dt != DType::C64 || int(n) < kTcMinQubits) return NQPU_MODE_TILED;
  PlanStats ts;
  if (!tc_plan_stats(ops, int(n), dt, &ts)) return NQPU_MODE_TILED;
  double work = 0.0;
  for (const Op& op : ops) {
    switch (op.kind) {
      case OP_U1: work += op.nctrl ? 0.15 : 0.071; break;
      case OP_U2: work += 0.30; break;
      case OP_D1:
      case OP_D2:
      case OP_PH: work += 0.011; break;
      default: break;  // OP_X1, OP_SW
    }
  }
  const double unit = 2.0 * std::ldexp(8.0, int(n)) / 6.5e6;  // 2 S bytes at 6.5 TB/s, in microseconds
  const double xp = double(ts.passes);
  const double tensor = unit * (1.013 * xp + 0.139 * double(ts.stages)) + 16.8 * xp + 34.0;
  auto tiled = [&](const TilePlan& p) {
    const double tp = double(p.stats.passes), st = double(p.stats.stages);
    return unit * (0.80 * tp + 0.069 * st + work) + 11.2 * tp + 1.1 * st;
  };
  // The larger of the plan's two tile sizes shortens the tiled estimate by a sixth
  // at most (27-qubit phase estimation, 7 passes instead of 10), so where
  // the tensor passes win by a fifth its plan is not built (26-qubit
  // brickwork: this choice 446 us of host time, 261 without it).
  TilePlan tp;
  std::string err;
  if (!build_tile_plan_for(ops, int(n), dt, &tp, &err, [&](const TilePlan& p) { return tensor < 0.8 * tiled(p); }))
    return NQPU_MODE_TENSOR;
  if (tensor < tiled(tp)) return NQPU_MODE_TENSOR;
  if (plan) *plan = std::move(tp);
  return NQPU_MODE_TILED;
}

static std::vector<Op> segment_ops(const CircuitImpl* c, const Segment& seg) {
  return lower_circuit(std::vector<GateRec>(c->gates.begin() + long(seg.begin), c->gates.begin() + long(seg.end)));
}

bool circuit_plan_stats(const CircuitImpl* c, uint32_t n, DType dt, int mode, PlanStats* out) {
  *out = PlanStats{};
  for (const Segment& seg : circuit_segments(c->gates)) {
    DevicePlan p;
    PlanStats st;
    if (mode == NQPU_MODE_AUTO) {
      if (seg.begin == seg.end) continue;
      const int m = auto_mode_for(segment_ops(c, seg), n, dt);
      CircuitImpl one;
      one.n = c->n;
      one.gates.assign(c->gates.begin() + long(seg.begin), c->gates.begin() + long(seg.end));
      if (!circuit_plan_stats(&one, n, dt, m, &st)) return false;
      out->passes += st.passes;
      out->ops += st.ops;
      out->stages += st.stages;
      out->upload_bytes += st.upload_bytes;
      continue;
    }
    if (mode == NQPU_MODE_FUSED || mode == NQPU_MODE_TENSOR) {
      p.ops = lower_circuit(std::vector<GateRec>(c->gates.begin() + long(seg.begin), c->gates.begin() + long(seg.end)));
      const bool ok = mode == NQPU_MODE_FUSED ? fused_plan_stats(p.ops, int(n), dt, &st)
                                              : tc_plan_stats(p.ops, int(n), dt, &st);
      if (!ok) return false;
    } else {
      if (!plan_host(c, seg, n, dt, mode, nullptr, &p)) return false;
      st = p.stats;
    }
    out->passes += st.passes;
    out->ops += st.ops;
    out->stages += st.stages;
    out->upload_bytes += st.upload_bytes;
  }
  return true;
}

static cudaError_t mark(std::vector<cudaEvent_t>* ev, cudaStream_t st) {
  if (!ev) return cudaSuccess;
  cudaEvent_t e;
  cudaError_t r = cudaEventCreate(&e);
  if (r != cudaSuccess) return r;
  ev->push_back(e);
  return cudaEventRecord(e, st);
}

static cudaError_t segment_run(CircuitImpl* c, const Segment& seg, int si, StateImpl* s, int mode,
                               std::vector<cudaEvent_t>* events);

cudaError_t circuit_run(CircuitImpl* c, StateImpl* s, int mode, std::vector<cudaEvent_t>* events,
                        std::vector<uint32_t>* outcomes) {
  std::lock_guard<std::mutex> lk(c->mu);
  const std::vector<Segment> segs = circuit_segments(c->gates);
  // measurements are queued like every other launch; their results gather in
  // pinned memory and are read when it is full and at the end
  constexpr size_t kSlots = (kSmallDoubles - kSmallTable) / 2;
  size_t queued = 0;
  auto drain = [&]() {
    const cudaError_t e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return e;
    for (size_t i = 0; i < queued; ++i) outcomes->push_back(uint32_t(s->h_small[kSmallTable + 2 * i]));
    queued = 0;
    return cudaSuccess;
  };
  // no error leaves a kernel behind that still writes there: the next call stages
  // its own tables in the same memory
  auto fail = [&](cudaError_t e) {
    if (queued) drain();
    return e;
  };
  for (size_t si = 0; si < segs.size(); ++si) {
    const Segment& seg = segs[si];
    cudaError_t e = segment_run(c, seg, int(si), s, mode, events);
    if (e != cudaSuccess) return fail(e);
    if (seg.mid < 0) break;
    const GateRec& g = c->gates[size_t(seg.mid)];
    // OpenQASM reset: measure (one RNG draw) and flip the qubit back to |0>
    // when it came out 1 (the state API's nqpu_gate_reset_qubit keeps the
    // reference's projection, GateOperations::reset_qubit)
    double* res = nullptr;
    if (g.code == G_MEASURE && outcomes) {
      if (queued == kSlots && (e = drain()) != cudaSuccess) return e;
      res = s->h_small + kSmallTable + 2 * queued;
    }
    if ((e = state_queue_measure(s, uint32_t(g.q[0]), g.code == G_RESET, res)) != cudaSuccess) return fail(e);
    if (res) ++queued;
  }
  if (queued) return drain();
  return cudaSuccess;
}

static cudaError_t segment_run(CircuitImpl* c, const Segment& seg, int si, StateImpl* s, int mode,
                               std::vector<cudaEvent_t>* events) {
  if (seg.begin == seg.end) return cudaSuccess;
  TilePlan ready;
  if (mode == NQPU_MODE_AUTO) {
    CircuitImpl::AutoMode& am = c->auto_modes[std::make_tuple(s->n, int(s->dt), si)];
    if (am.version != c->version || am.tile_cfg != tile_config_get(s->dt))
      am = {c->version, tile_config_get(s->dt), auto_mode_for(segment_ops(c, seg), s->n, s->dt, &ready)};
    mode = am.mode;
  }
  const int effective = (mode == NQPU_MODE_TILED && int(s->n) < tile_min_qubits(s->dt)) ? int(NQPU_MODE_PERGATE) : mode;
  const auto key = std::make_tuple(s->n, int(s->dt), effective, si);
  DevicePlan*& p = c->plans[key];
  // rebuild when the circuit changed or the tiled kernel's tile size did
  if (p && (p->version != c->version || (effective == NQPU_MODE_TILED && p->tile_cfg != tile_config_get(s->dt)))) {
    cudaStreamSynchronize(s->stream);
    plan_free(p);
    p = nullptr;
  }
  if (!p) {
    p = new DevicePlan();
    p->tile = std::move(ready);
    if (!plan_host(c, seg, s->n, s->dt, effective, s->stream, p)) {
      plan_free(p);
      p = nullptr;
      return cudaErrorInvalidValue;
    }
    if (effective == NQPU_MODE_TILED) {
      const std::vector<ProgWord>& prog = p->tile.prog;
      cudaError_t e = upload_table(reinterpret_cast<void**>(&p->d_prog), prog.data(), prog.size() * sizeof(ProgWord), s->stream);
      if (e != cudaSuccess) {
        plan_free(p);
        p = nullptr;
        return e;
      }
    }
    p->version = c->version;
  }
  cudaError_t e = mark(events, s->stream);
  if (e != cudaSuccess) return e;
  if (effective == NQPU_MODE_PERGATE) {
    for (const Op& op : p->ops) {
      if ((e = launch_pergate(s->dt, s->amp, int(s->n), op, s->next_sweep(), s->stream, device_sms())) != cudaSuccess) return e;
      if ((e = mark(events, s->stream)) != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  if (effective == NQPU_MODE_FUSED) {
    e = fused_run(p->fused, s, events);
    if (e != cudaSuccess) return e;
    return state_run_error(s);  // bounded-wait expiry flag
  }
  if (effective == NQPU_MODE_TENSOR) {
    e = tc_run(p->tc, s, events);
    if (e != cudaSuccess) return e;
    return state_run_error(s);  // bounded-wait expiry flag
  }
  for (size_t i = 0; i < p->tile.passes.size(); ++i) {
    e = launch_tile_pass(s->dt, s->amp, p->tile.passes[i], p->d_prog, s->stream, device_sms());
    if (e != cudaSuccess) return e;
    if ((e = mark(events, s->stream)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace nqpu
