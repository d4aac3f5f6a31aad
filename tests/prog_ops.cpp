// Test infrastructure: lowered ops that no gate of the interface lowers to, through
// the stage program compiler and the interpreter of prog_emulator.cpp.
#include "prog_emulator.cpp"

// A 2x2 on qubit `target` controlled by the qubits of `ctrl` (three at most), between
// two layers of its own, on a register of the stage's own bits (5 qubits complex64, 4
// complex128): the largest amplitude error against the op applied directly, or a
// negative number where the program does not run.
template <typename Real>
static double controlled(int target, uint32_t ctrl) {
  constexpr bool F32 = sizeof(Real) == 4;
  const int n = F32 ? 5 : 4;
  std::vector<Op> ops;
  auto u = [&](int t, uint32_t cm, double x) {
    Op o;
    o.kind = OP_U1;
    o.t0 = int8_t(t);
    for (int q = 0; q < n; ++q)
      if ((cm >> q) & 1) o.ctrl[o.nctrl++] = int8_t(q);
    o.m[0] = std::cos(x);
    o.m[1] = -std::sin(x) * std::polar(1.0, 0.7);
    o.m[2] = std::sin(x) * std::polar(1.0, 0.4);
    o.m[3] = std::cos(x) * std::polar(1.0, 1.1);
    ops.push_back(o);
  };
  for (int q = 0; q < n; ++q) u(q, 0, 0.3 + 0.2 * q);
  u(target, ctrl, 0.9);
  for (int q = 0; q < n; ++q) u(q, 0, 1.2 - 0.1 * q);
  std::vector<cd> a(size_t(1) << n), b;
  for (size_t i = 0; i < a.size(); ++i) a[i] = std::polar(1.0 / std::sqrt(double(a.size())), double(i * i));
  b = a;
  for (const Op& o : ops)
    for (size_t i = 0; i < b.size(); ++i) {
      const size_t t = size_t(1) << o.t0;
      if ((i & t) || (i & o.ctrl_mask()) != o.ctrl_mask()) continue;
      const cd x = b[i], y = b[i | t];
      b[i] = o.m[0] * x + o.m[1] * y;
      b[i | t] = o.m[2] * x + o.m[3] * y;
    }
  TilePlan plan;
  std::string err;
  const std::vector<Op> carried = carry_phases(ops);
  if (!build_tile_plan(carried, n, F32 ? DType::C64 : DType::C128, 12, &plan, &err) || plan.stages.size() != 1) return -1;
  build_tile_prog(carried, &plan);
  const ProgWord* w = plan.prog.data() + kStageTabWords / 4;
  if (run_words<Real>(w + plan.stages[0].prog_begin, w + plan.stages[0].prog_end, a, 0)) return -2;
  double e = 0;
  for (size_t i = 0; i < a.size(); ++i) e = std::max(e, std::abs(a[i] - b[i]));
  return e;
}

// What the tile kernel cannot do: a 2x2 with more than one register control.
template <typename Real>
static int records_fit(int target, uint32_t ctrl) {
  const int n = sizeof(Real) == 4 ? 5 : 4;
  Op o;
  o.kind = OP_U1;
  o.t0 = int8_t(target);
  for (int q = 0; q < n; ++q)
    if ((ctrl >> q) & 1) o.ctrl[o.nctrl++] = int8_t(q);
  o.m[0] = o.m[3] = 0.6;
  o.m[1] = -0.8;
  o.m[2] = 0.8;
  TilePlan plan;
  std::string err;
  if (!build_tile_plan({o}, n, n == 5 ? DType::C64 : DType::C128, 12, &plan, &err)) return -1;
  build_tile_prog({o}, &plan);
  const StageRec& S = plan.stages[0];
  int records = 0;
  for (int i = S.prog_begin; i < S.prog_end; ++i) {
    const ProgWord& h = plan.prog[size_t(kStageTabWords / 4 + i)];
    i += int(h.w[0] >> 16) - 1;
    if ((h.w[0] & 0xFF) != TC_OP) continue;
    ++records;
    const uint32_t creg = h.w[1] >> 16;
    if (((h.w[0] >> 8) & 0xFF) == OP_U1 && (creg & (creg - 1))) return -2;
  }
  return records;
}

extern "C" double controlled_2x2(int c64, int target, int ctrl) {
  return c64 ? controlled<float>(target, uint32_t(ctrl)) : controlled<double>(target, uint32_t(ctrl));
}
extern "C" int controlled_records(int c64, int target, int ctrl) {
  return c64 ? records_fit<float>(target, uint32_t(ctrl)) : records_fit<double>(target, uint32_t(ctrl));
}
