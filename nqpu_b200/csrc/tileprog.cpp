// Compiler of the tiled passes' stage programs (encoding: tileprog.h).
#include "tileprog.h"
#include <cmath>
#include <cstring>

namespace nqpu {
namespace {

struct Entry {
  uint32_t mask;
  cplx p;
};
// Pending phase on the register amplitudes with bits A set.
struct Phase {
  bool used = false;
  cplx uniform{1.0, 0.0};
  std::vector<Entry> list;
  bool trivial() const { return list.empty() && uniform == cplx(1.0, 0.0); }
  bool signs() const {  // only factors of +1 and -1
    if (uniform != cplx(1.0, 0.0) && uniform != cplx(-1.0, 0.0)) return false;
    for (const Entry& e : list)
      if (e.p != cplx(-1.0, 0.0)) return false;
    return true;
  }
};

struct Instr {
  enum Kind { DENSE, PHASE, PAIR, LEGACY } kind = DENSE;
  int bit = 0;         // DENSE, PAIR
  uint32_t cnr = 0;    // DENSE
  cplx m[4];           // DENSE
  uint32_t A = 0;      // PHASE
  Phase a, b;          // PHASE: a; PAIR: all amplitudes, amplitudes with `bit`
  size_t op = 0;       // LEGACY: index into the plan's ops
};

// Angle in 2^-32 turns of a unit complex number.
uint32_t turns(cplx p) {
  const double t = std::atan2(p.imag(), p.real()) / 6.283185307179586476925;
  return uint32_t(int64_t(std::llround(t * 4294967296.0)));
}

class Writer {
 public:
  explicit Writer(std::vector<ProgWord>* out, bool f32) : out_(out), f32_(f32) {}
  size_t header(uint32_t code, uint32_t y = 0) {
    begin_ = out_->size();
    out_->push_back(ProgWord{{code, y, 0, 0}});
    return begin_;
  }
  void end() { (*out_)[begin_].w[0] |= uint32_t(out_->size() - begin_) << 16; }
  ProgWord& head() { return (*out_)[begin_]; }
  void reals(const double* v, int n) {
    if (f32_) {
      std::vector<float> f(v, v + n);
      bytes(f.data(), sizeof(float) * size_t(n));
    } else {
      bytes(v, sizeof(double) * size_t(n));
    }
  }
  void bytes(const void* p, size_t n) {
    const size_t w = (n + 15) / 16, at = out_->size();
    out_->resize(at + w, ProgWord{{0, 0, 0, 0}});
    std::memcpy(&(*out_)[at], p, n);
  }
  void list(const std::vector<Entry>& l) {
    if (f32_) {
      std::vector<uint32_t> v;
      for (const Entry& e : l) { v.push_back(e.mask); v.push_back(turns(e.p)); }
      if (!v.empty()) bytes(v.data(), v.size() * 4);
    } else {
      for (const Entry& e : l) {
        out_->push_back(ProgWord{{e.mask, 0, 0, 0}});
        const double v[2] = {e.p.real(), e.p.imag()};
        reals(v, 2);
      }
    }
  }

 private:
  std::vector<ProgWord>* out_;
  bool f32_;
  size_t begin_ = 0;
};

template <typename Real>
class StageCompiler {
 public:
  StageCompiler(const std::vector<Op>& ops, const TilePlan& plan, const std::vector<TileOp<Real>>& enc)
      : ops_(ops), plan_(plan), enc_(enc) {}

  // Compile stage S; `global` is the phase common to all amplitudes, carried from
  // stage to stage and applied by the last one.
  void run(const StageRec& S, bool last, cplx* global, std::vector<ProgWord>* out) {
    code_.clear();
    for (Phase& p : pend_) p = Phase();
    for (int& o : open_) o = -1;
    for (int o = S.op_begin; o < S.op_end; ++o) add(size_t(o));
    *global *= pend_[0].uniform;
    pend_[0].uniform = last ? *global : cplx(1.0, 0.0);
    finish();
    emit(out);
  }

 private:
  static constexpr int kBits = sizeof(Real) == 4 ? 5 : 4;

  void phase(uint32_t A, uint32_t B, cplx p) {
    Phase& P = pend_[A];
    P.used = true;
    if (B == 0) { P.uniform *= p; return; }
    for (size_t i = 0; i < P.list.size(); ++i)
      if (P.list[i].mask == B) {
        P.list[i].p *= p;
        if (P.list[i].p == cplx(1.0, 0.0)) P.list.erase(P.list.begin() + long(i));
        return;
      }
    P.list.push_back(Entry{B, p});
  }

  // Emit the pending phases that do not commute with a dense op on bits `t`.
  void flush(uint32_t t) {
    for (uint32_t A = 1; A < (1u << kBits); ++A) {
      if (!(A & t) || !pend_[A].used) continue;
      put(A, pend_[A]);
      pend_[A] = Phase();
    }
  }

  void put(uint32_t A, const Phase& P) {
    if (P.trivial()) return;
    // a constant phase on one bit goes into the complex matrix before it
    if ((A & (A - 1)) == 0 && A != 0 && P.list.empty()) {
      const int o = open_[ctz(A)];
      if (o >= 0 && code_[size_t(o)].cnr == 0 && generic(code_[size_t(o)].m)) {
        code_[size_t(o)].m[2] *= P.uniform;
        code_[size_t(o)].m[3] *= P.uniform;
        return;
      }
    }
    for (int b = 0; b < kBits; ++b)
      if ((A >> b) & 1) open_[b] = -1;
    Instr I;
    I.kind = Instr::PHASE;
    I.A = A;
    I.a = P;
    code_.push_back(I);
  }

  // Stage end: what is left; the phase on all amplitudes joins a one-bit phase.
  void finish() {
    const Phase all = pend_[0];
    int join = -1;
    if (!all.trivial())
      for (int b = 0; b < kBits && join < 0; ++b) {
        const Phase& P = pend_[1u << b];
        if (P.used && !P.trivial() && !P.signs()) join = b;
      }
    for (uint32_t A = 1; A < (1u << kBits); ++A) {
      if (!pend_[A].used || (join >= 0 && A == (1u << join))) continue;
      put(A, pend_[A]);
    }
    if (join >= 0) {
      Instr I;
      I.kind = Instr::PAIR;
      I.bit = join;
      I.a = all;
      I.b = pend_[1u << join];
      code_.push_back(I);
    } else {
      put(0, all);
    }
  }

  static int ctz(uint32_t v) { return __builtin_ctz(v); }
  static bool real(const cplx* m) {
    return m[0].imag() == 0 && m[1].imag() == 0 && m[2].imag() == 0 && m[3].imag() == 0;
  }
  static bool cross(const cplx* m) {
    return m[0].imag() == 0 && m[1].real() == 0 && m[2].real() == 0 && m[3].imag() == 0;
  }
  static bool generic(const cplx* m) { return !real(m) && !cross(m); }

  void add(size_t oi) {
    const TileOp<Real>& t = enc_[oi];
    const Op& o = ops_[size_t(plan_.op_src[oi])];
    switch (t.kind) {
      case OP_PH:
        phase(t.creg, t.cnr, o.m[0]);
        return;
      case OP_D1: {
        const uint32_t a = t.dreg0 != 0xFF ? 1u << t.dreg0 : 0u;
        phase(t.creg, t.cnr, o.m[0]);
        phase(t.creg | a, t.cnr | t.dv0, o.m[1] / o.m[0]);
        return;
      }
      case OP_D2: {
        const uint32_t a = t.dreg0 != 0xFF ? 1u << t.dreg0 : 0u, b = t.dreg1 != 0xFF ? 1u << t.dreg1 : 0u;
        phase(t.creg, t.cnr, o.m[0]);
        phase(t.creg | a, t.cnr | t.dv0, o.m[1] / o.m[0]);
        phase(t.creg | b, t.cnr | t.dv1, o.m[2] / o.m[0]);
        phase(t.creg | a | b, t.cnr | t.dv0 | t.dv1, (o.m[3] * o.m[0]) / (o.m[1] * o.m[2]));
        return;
      }
      case OP_U1:
        if (t.creg == 0) { dense(t.rb0, t.cnr, o.m); return; }
        break;
      default:
        break;
    }
    uint32_t touched = 1u << t.rb0;
    if (t.kind == OP_U2 || t.kind == OP_SW) touched |= 1u << t.rb1;
    flush(touched);
    // the op reads its register controls: it stays after what wrote them
    touched |= t.creg;
    for (int b = 0; b < kBits; ++b)
      if ((touched >> b) & 1) open_[b] = -1;
    Instr I;
    I.kind = Instr::LEGACY;
    I.op = oi;
    code_.push_back(I);
  }

  void dense(int b, uint32_t cnr, const cplx* m) {
    // phases on this bit alone and constant: into the matrix where that makes
    // the product no dearer (it is complex already, or the gate before it on
    // this bit is still open to take it)
    cplx M[4] = {m[0], m[1], m[2], m[3]};
    Phase& P = pend_[1u << b];
    const bool merge = open_[b] >= 0 && code_[size_t(open_[b])].cnr == cnr;
    bool others = false;
    for (uint32_t A = 1; A < (1u << kBits); ++A)
      if ((A >> b) & 1 && A != (1u << b) && pend_[A].used && !pend_[A].trivial()) others = true;
    if (P.used && P.list.empty() && cnr == 0 && (generic(M) || (merge && !others))) {
      M[1] *= P.uniform;
      M[3] *= P.uniform;
      P = Phase();
    }
    if (merge && !others && (!P.used || P.trivial())) {
      cplx* p = code_[size_t(open_[b])].m;
      const cplx r[4] = {M[0] * p[0] + M[1] * p[2], M[0] * p[1] + M[1] * p[3],
                         M[2] * p[0] + M[3] * p[2], M[2] * p[1] + M[3] * p[3]};
      std::memcpy(p, r, sizeof(r));
      return;
    }
    flush(1u << b);
    Instr I;
    I.kind = Instr::DENSE;
    I.bit = b;
    I.cnr = cnr;
    for (int i = 0; i < 4; ++i) I.m[i] = M[i];
    open_[b] = int(code_.size());
    code_.push_back(I);
  }

  void emit(std::vector<ProgWord>* out) {
    constexpr bool f32 = sizeof(Real) == 4;
    Writer W(out, f32);
    for (const Instr& I : code_) {
      switch (I.kind) {
        case Instr::DENSE: {
          if (real(I.m)) {
            const double v[4] = {I.m[0].real(), I.m[1].real(), I.m[2].real(), I.m[3].real()};
            W.header(TC_R + uint32_t(I.bit), I.cnr);
            W.reals(v, 4);
          } else if (cross(I.m)) {
            const double v[4] = {I.m[0].real(), I.m[1].imag(), I.m[2].imag(), I.m[3].real()};
            W.header(TC_X + uint32_t(I.bit), I.cnr);
            W.reals(v, 4);
          } else {
            double v[8];
            for (int i = 0; i < 4; ++i) { v[2 * i] = I.m[i].real(); v[2 * i + 1] = I.m[i].imag(); }
            W.header(TC_G + uint32_t(I.bit), I.cnr);
            W.reals(v, 8);
          }
          break;
        }
        case Instr::PHASE: {
          const Phase& P = I.a;
          const double u[2] = {P.uniform.real(), P.uniform.imag()};
          if (P.signs()) {
            W.header(TC_SG + I.A, uint32_t(P.list.size()));
            W.head().w[2] = P.uniform.real() < 0 ? 1u : 0u;
            std::vector<uint32_t> v;
            for (const Entry& e : P.list) v.push_back(e.mask);
            while (v.size() % 4) v.push_back(~0u);  // never matched: counted off by header.y
            if (!v.empty()) W.bytes(v.data(), v.size() * 4);
          } else if (f32 && P.list.empty()) {
            W.header(TC_PU + I.A);
            const float f[2] = {float(u[0]), float(u[1])};
            std::memcpy(&W.head().w[2], f, 8);
          } else {
            W.header(TC_PH + I.A, uint32_t(P.list.size()));
            if (f32) W.head().w[2] = turns(P.uniform);
            else W.reals(u, 2);
            W.list(P.list);
          }
          break;
        }
        case Instr::PAIR: {
          W.header(TC_D + uint32_t(I.bit), uint32_t(I.a.list.size()) | uint32_t(I.b.list.size()) << 16);
          if (f32) {
            W.head().w[2] = turns(I.a.uniform);
            W.head().w[3] = turns(I.b.uniform);
          } else {
            const double u[4] = {I.a.uniform.real(), I.a.uniform.imag(), I.b.uniform.real(), I.b.uniform.imag()};
            W.reals(u, 4);
          }
          W.list(I.a.list);
          W.list(I.b.list);
          break;
        }
        case Instr::LEGACY:
          W.header(TC_LEG);
          W.bytes(&enc_[I.op], sizeof(TileOp<Real>));
          break;
      }
      W.end();
    }
  }

  const std::vector<Op>& ops_;
  const TilePlan& plan_;
  const std::vector<TileOp<Real>>& enc_;
  std::vector<Instr> code_;
  Phase pend_[32];
  int open_[5];
};

// Shared-memory slot of vector u (the kernels' swz).
uint32_t swz(uint32_t u) {
  const uint32_t w = u >> 3, f = w ^ (w >> 3) ^ (w >> 6) ^ (w >> 9) ^ (w >> 12);
  return u ^ (f & 7u);
}

void stage_tab(const StageRec& S, int vb, uint32_t (&t)[kStageTabWords]) {
  uint32_t s[4];
  for (int i = 0; i < 4; ++i) s[i] = swz(1u << (S.rpos[i] - vb));
  auto regslot = [&](uint32_t m) {
    uint32_t x = 0;
    for (int i = 0; i < 4; ++i)
      if ((m >> (vb + i)) & 1u) x ^= s[i];
    return x;
  };
  auto half = [&](uint32_t m) { return vb == 1 ? (m & 1u) : 0u; };
  t[StageTab::HB] = 0;
  for (int i = 0; i < 4; ++i) {
    const uint32_t m = uint32_t(S.scol[vb + i]);
    t[StageTab::S + i] = s[i];
    t[StageTab::CW + i] = regslot(m);
    t[StageTab::HB] |= half(m) << i;
  }
  const uint32_t mz = vb == 1 ? uint32_t(S.scol[0]) : 1u;
  t[StageTab::MZ] = mz;
  t[StageTab::CZ] = regslot(mz);
  t[StageTab::HZ] = half(mz);
  t[StageTab::WS] = regslot(uint32_t(S.sbx));
  t[StageTab::WH] = half(uint32_t(S.sbx));
  t[StageTab::NC] = uint32_t(S.ncond);
  t[StageTab::OB] = uint32_t(S.prog_begin);
  t[StageTab::OE] = uint32_t(S.prog_end);
  for (int i = 0; i < kMaxCondPerm; ++i) {
    const uint32_t w = uint32_t(S.cond_w[i]);
    t[StageTab::CC + i] = S.cond_cnr[i];
    t[StageTab::CS + i] = regslot(w);
    t[StageTab::CH + i] = half(w);
  }
  for (int v = 0; v < 16; ++v) {
    uint32_t lo = 0, hi = 0;
    for (int j = 0; j < 4; ++j) {
      if (j < S.n_tbits && ((v >> j) & 1)) lo |= 1u << S.tpos[j];
      if (j + 4 < S.n_tbits && ((v >> j) & 1)) hi |= 1u << S.tpos[j + 4];
    }
    t[StageTab::UL + v] = lo;
    t[StageTab::UH + v] = hi;
    t[StageTab::SL + v] = swz(lo);
    t[StageTab::SH + v] = swz(hi);
  }
}

template <typename Real>
void compile(const std::vector<Op>& ops, TilePlan* plan, const std::vector<TileOp<Real>>& enc) {
  StageCompiler<Real> C(ops, *plan, enc);
  cplx global(1.0, 0.0);
  const size_t last = plan->stages.empty() ? 0 : plan->stages.size() - 1;
  for (PassRec& P : plan->passes) {
    P.prog_begin = int32_t(plan->prog.size());
    const size_t tabs = plan->prog.size(), base = tabs + size_t(P.stage_end - P.stage_begin) * (kStageTabWords / 4);
    plan->prog.resize(base, ProgWord{{0, 0, 0, 0}});
    for (int s = P.stage_begin; s < P.stage_end; ++s) {
      StageRec& S = plan->stages[size_t(s)];
      S.prog_begin = int32_t(plan->prog.size() - base);
      C.run(S, size_t(s) == last, &global, &plan->prog);
      S.prog_end = int32_t(plan->prog.size() - base);
      uint32_t tab[kStageTabWords] = {};
      stage_tab(S, plan->dt == DType::C64 ? 1 : 0, tab);
      std::memcpy(static_cast<void*>(plan->prog.data() + tabs + size_t(s - P.stage_begin) * (kStageTabWords / 4)), tab,
                  sizeof(tab));
    }
    P.prog_words = int32_t(plan->prog.size() - tabs);
  }
}

}  // namespace

void build_tile_prog(const std::vector<Op>& ops, TilePlan* plan) {
  plan->prog.clear();
  if (plan->dt == DType::C64) compile<float>(ops, plan, plan->ops_f);
  else compile<double>(ops, plan, plan->ops_d);
  plan->stats.upload_bytes = plan->passes.size() * sizeof(PassRec) + plan->prog.size() * sizeof(ProgWord);
}

}  // namespace nqpu
