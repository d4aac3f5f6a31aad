// Compiler of the tiled passes' stage programs (encoding: tileprog.h).
#include "tileprog.h"
#include <algorithm>
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
  void clear() {  // keeps the list's memory
    used = false;
    uniform = cplx(1.0, 0.0);
    list.clear();
  }
  bool trivial() const { return list.empty() && uniform == cplx(1.0, 0.0); }
  bool signs() const {  // only factors of +1 and -1
    if (uniform != cplx(1.0, 0.0) && uniform != cplx(-1.0, 0.0)) return false;
    for (const Entry& e : list)
      if (e.p != cplx(-1.0, 0.0)) return false;
    return true;
  }
};

// An op of a stage, or a part of one, before scheduling.
struct Item {
  enum Kind { PHASE, ROT, CROSS, FLIP, GENERIC, RECORD } kind = PHASE;
  uint32_t diag = 0, dense = 0;  // register bits it reads (commutes with phases) / changes
  uint32_t cnr = 0;              // virtual-index mask: a phase's condition, a 2x2's control
  cplx m[4];                     // PHASE: m[0]; GENERIC: the matrix
  double t = 0, s = 0;           // ROT, CROSS
  size_t op = 0;                 // RECORD: index into the plan's ops
};

// Angle in 2^-32 turns of a unit complex number.
uint32_t turns(cplx p) {
  const double t = std::atan2(p.imag(), p.real()) / 6.283185307179586476925;
  return uint32_t(int64_t(std::llround(t * 4294967296.0)));
}

class Writer {
 public:
  explicit Writer(std::vector<ProgWord>* out, bool f32) : out_(out), f32_(f32) {}
  size_t header(uint32_t code, uint32_t arg, uint32_t y = 0) {
    begin_ = out_->size();
    out_->push_back(ProgWord{{code | arg << 8, y, 0, 0}});
    return begin_;
  }
  void end() { (*out_)[begin_].w[0] |= uint32_t(out_->size() - begin_) << 16; }
  ProgWord& head() { return (*out_)[begin_]; }  // valid until more is written
  void reals(const double* v, int n) {  // at most 64
    if (f32_) {
      float f[64];
      for (int i = 0; i < n; ++i) f[i] = float(v[i]);
      bytes(f, sizeof(float) * size_t(n));
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
      for (size_t i = 0; i < l.size(); i += 2) {
        const bool two = i + 1 < l.size();
        out_->push_back(ProgWord{{l[i].mask, turns(l[i].p), two ? l[i + 1].mask : 0u, two ? turns(l[i + 1].p) : 0u}});
      }
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
      : ops_(ops), plan_(plan), enc_(enc), W_(nullptr, sizeof(Real) == 4) {}

  // Compile stage S; `global` is the phase common to all amplitudes, carried from
  // stage to stage and applied by the last one.
  void run(const StageRec& S, bool last, cplx* global, std::vector<ProgWord>* out) {
    W_ = Writer(out, sizeof(Real) == 4);
    global_ = global;
    final_ = false;
    items_.clear();
    dense_bits_ = 0;
    for (Phase& p : pend_) p.clear();
    used_ = 0;
    for (bool& h : have_) h = false;
    for (int o = S.op_begin; o < S.op_end; ++o) add(size_t(o));
    for (int b = 0; b < kBits; ++b) settle(b);
    schedule();
    *global *= pend_[0].uniform;
    pend_[0].uniform = last ? *global : cplx(1.0, 0.0);
    final_ = last;
    finish();
  }

 private:
  static constexpr bool kF32 = sizeof(Real) == 4;
  static constexpr int kBits = kF32 ? 5 : 4;
  static constexpr uint32_t kAll = 1u << kBits;

  // ---- ops to items -------------------------------------------------------
  // 2x2s on a register bit and constant phases on it alone multiply up in acc_
  // until something that does not commute with them arrives.
  void phase(uint32_t A, uint32_t B, cplx p) {
    if ((A & (A - 1)) == 0 && A != 0 && B == 0 && have_[ctz(A)]) {
      acc_[ctz(A)][2] *= p;
      acc_[ctz(A)][3] *= p;
      return;
    }
    for (int b = 0; b < kBits; ++b)
      if ((A >> b) & 1) settle(b);
    push_phase(A, B, p);
  }
  void push_phase(uint32_t A, uint32_t B, cplx p) {
    if (p == cplx(1.0, 0.0)) return;
    if (!(A & dense_bits_)) {  // nothing to wait for
      pend(A, B, p);
      return;
    }
    Item I;
    I.diag = A;
    I.cnr = B;
    I.m[0] = p;
    items_.push_back(I);
  }

  void push_dense(const Item& I) {
    dense_bits_ |= I.dense;
    items_.push_back(I);
  }

  void settle(int b) {
    if (!have_[b]) return;
    have_[b] = false;
    dense(b, 0, acc_[b]);
  }

  // Magnitudes and quotients of unitaries' entries and phases.  The operands of
  // complex64 programs are rounded to 2^-24, so hypot, the full complex division and
  // (join_constant) an angle per table entry buy nothing there: a circuit that runs
  // once pays for its program (17-qubit brickwork, 375 gates: build_tile_prog 165 ->
  // 95 us, 77 with phases that wait for nothing taken at once; complex128 keeps
  // them, its results are 1e-15 off).
  static double mag(cplx z) { return kF32 ? std::sqrt(std::norm(z)) : std::abs(z); }
  static cplx unit(cplx z) { return z / mag(z); }
  static cplx quot(cplx z, cplx w) { return kF32 ? z * std::conj(w) / std::norm(w) : z / w; }
  static cplx over(cplx z, cplx w) { return kF32 ? z * std::conj(w) : z / w; }  // w a unit

  // A 2x2 as items: phase x rotation x phase where it is unitary, else as it is.
  void dense(int b, uint32_t cnr, const cplx* m) {
    Item I;
    I.dense = 1u << b;
    I.cnr = cnr;
    const double eps = 1e-12;
    const bool unitary = cnr == 0 && std::abs(std::norm(m[0]) + std::norm(m[2]) - 1.0) < eps &&
                         std::abs(std::norm(m[1]) + std::norm(m[3]) - 1.0) < eps &&
                         std::norm(std::conj(m[0]) * m[1] + std::conj(m[2]) * m[3]) < eps * eps;
    if (!unitary) {
      I.kind = Item::GENERIC;
      for (int i = 0; i < 4; ++i) I.m[i] = m[i];
      push_dense(I);
      return;
    }
    const double c = mag(m[0]), s = mag(m[2]);
    if (c < kFlip) {  // Y, RX(pi), RY(pi): the amplitudes change places, with phases
      I.kind = Item::FLIP;
      push_dense(I);
      push_phase(0, 0, unit(m[1]));
      push_phase(1u << b, 0, clean(unit(quot(m[2], m[1]))));
      return;
    }
    // RX: cos and -i sin
    if (m[0].imag() == 0 && m[3].imag() == 0 && m[1].real() == 0 && m[2].real() == 0 && m[0].real() == m[3].real() &&
        m[1].imag() == m[2].imag()) {
      const double sg = m[0].real() < 0 ? -1.0 : 1.0;  // |phi| <= pi/2 up to a common sign
      push_phase(0, 0, cplx(sg, 0.0));
      shears(sg * m[0].real(), -sg * m[1].imag(), &I);
      I.kind = Item::CROSS;
      if (I.s != 0.0) push_dense(I);
      return;
    }
    const cplx one(1.0, 0.0);
    if (s < kTiny) {  // a phase
      push_phase(0, 0, unit(m[0]));
      push_phase(1u << b, 0, clean(unit(quot(m[3], m[0]))));
      return;
    }
    // e^{ia} diag(1, after) [[c, -s], [s, c]] diag(1, before)
    const cplx a = m[0] / c;
    // (`before` from the larger of the entries that fix it: a small off-diagonal
    // has no precise phase, and only its product with `after` matters then)
    const cplx after0 = over(m[2] / s, a);
    cplx after = unit(after0), before = unit(s > c ? over(-m[1] / s, a) : over(over(m[3] / c, a), after0));
    double sn = s;
    if (std::norm(after + one) < kTiny * kTiny) {  // a rotation the other way
      sn = -s;
      after = -after;
      before = -before;
    }
    push_phase(0, 0, a);
    push_phase(1u << b, 0, clean(before));
    shears(c, sn, &I);
    I.kind = Item::ROT;
    push_dense(I);
    push_phase(1u << b, 0, clean(after));
  }
  // A phase that is 1 or -1 up to the rounding of its making.
  static constexpr double kTiny = 1e-15;
  // |cos| below which a rotation is an exchange.  Three shears by a quarter turn add
  // either amplitude to the other and take it off again, which costs a small one its
  // digits beside a large one; leaving out less than half an ulp of the large one
  // does not cost more.
  static constexpr double kFlip = kF32 ? 1e-15 : 0x1p-53;
  static cplx clean(cplx p) {
    if (std::norm(p - cplx(1.0, 0.0)) < kTiny * kTiny) return cplx(1.0, 0.0);
    return std::norm(p + cplx(1.0, 0.0)) < kTiny * kTiny ? cplx(-1.0, 0.0) : p;
  }
  static void shears(double c, double s, Item* I) {  // c >= 0
    const double h = mag(cplx(c, s));
    I->t = (s / h) / (1.0 + c / h);
    I->s = s / h;
  }

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
        phase(t.creg | a, t.cnr | t.dv0, quot(o.m[1], o.m[0]));
        return;
      }
      case OP_D2: {
        const uint32_t a = t.dreg0 != 0xFF ? 1u << t.dreg0 : 0u, b = t.dreg1 != 0xFF ? 1u << t.dreg1 : 0u;
        phase(t.creg, t.cnr, o.m[0]);
        phase(t.creg | a, t.cnr | t.dv0, quot(o.m[1], o.m[0]));
        phase(t.creg | b, t.cnr | t.dv1, quot(o.m[2], o.m[0]));
        phase(t.creg | a | b, t.cnr | t.dv0 | t.dv1, quot(o.m[3] * o.m[0], o.m[1] * o.m[2]));
        return;
      }
      case OP_U1:
        if (t.creg != 0) break;
        if (t.cnr != 0) {
          settle(t.rb0);
          dense(t.rb0, t.cnr, o.m);
          return;
        }
        if (have_[t.rb0]) {
          const cplx* p = acc_[t.rb0];
          const cplx r[4] = {o.m[0] * p[0] + o.m[1] * p[2], o.m[0] * p[1] + o.m[1] * p[3],
                             o.m[2] * p[0] + o.m[3] * p[2], o.m[2] * p[1] + o.m[3] * p[3]};
          for (int i = 0; i < 4; ++i) acc_[t.rb0][i] = r[i];
        } else {
          have_[t.rb0] = true;
          for (int i = 0; i < 4; ++i) acc_[t.rb0][i] = o.m[i];
        }
        return;
      default:
        break;
    }
    Item I;
    I.kind = Item::RECORD;
    I.op = oi;
    I.dense = 1u << t.rb0;
    if (t.kind == OP_U2 || t.kind == OP_SW) I.dense |= 1u << t.rb1;
    I.diag = t.creg;
    for (int b = 0; b < kBits; ++b)
      if (((I.dense | I.diag) >> b) & 1) settle(b);
    push_dense(I);
  }

  // ---- scheduling ---------------------------------------------------------
  // Rounds of: take every phase that no earlier open dense item blocks, then emit
  // every dense item with nothing open before it on its bits.  Phases gather
  // as long as they can, so that a layer's join in one instruction.
  //
  // An item waits for the last dense item before it on each of its bits and, where
  // it is dense, for the items since then that read the bit; a round takes what
  // waits for nothing any more, in circuit order.  So the work is linear in the
  // items: walking all of them in every round took 580 ms for 18000 gates of an
  // Ising evolution on five qubits, which are one stage (now 9).
  void schedule() {
    const size_t n = items_.size();
    wait_.assign(n, 0);
    first_.assign(n, -1);
    edges_.clear();
    phases_.clear();
    dense_.clear();
    int last[kBits];
    for (int b = 0; b < kBits; ++b) {
      last[b] = -1;
      readers_[b].clear();
    }
    auto edge = [&](int from, int to) {
      edges_.push_back({to, first_[size_t(from)]});
      first_[size_t(from)] = int(edges_.size()) - 1;
      ++wait_[size_t(to)];
    };
    auto ready = [&](int i) { (items_[size_t(i)].kind == Item::PHASE ? phases_ : dense_).push_back(i); };
    for (int i = 0; i < int(n); ++i) {
      const Item& I = items_[size_t(i)];
      for (uint32_t w = I.diag | I.dense; w; w &= w - 1)
        if (last[ctz(w)] >= 0) edge(last[ctz(w)], i);
      for (uint32_t w = I.dense; w; w &= w - 1) {
        for (int r : readers_[ctz(w)]) edge(r, i);
        readers_[ctz(w)].clear();
        last[ctz(w)] = i;
      }
      for (uint32_t w = I.diag; w; w &= w - 1) readers_[ctz(w)].push_back(i);
      if (wait_[size_t(i)] == 0) ready(i);
    }
    auto release = [&](int i) {
      for (int e = first_[size_t(i)]; e >= 0; e = edges_[size_t(e)].next)
        if (--wait_[size_t(edges_[size_t(e)].to)] == 0) ready(edges_[size_t(e)].to);
    };
    for (;;) {
      std::sort(phases_.begin(), phases_.end());
      for (int i : phases_) {  // frees dense items only
        pend(items_[size_t(i)].diag, items_[size_t(i)].cnr, items_[size_t(i)].m[0]);
        release(i);
      }
      phases_.clear();
      if (dense_.empty()) break;
      batch_.swap(dense_);
      dense_.clear();
      std::sort(batch_.begin(), batch_.end());
      uint32_t bits = 0;
      for (int i : batch_) bits |= items_[size_t(i)].dense;
      flush(bits);
      emit_rotations(Item::ROT);
      emit_rotations(Item::CROSS);
      for (int i : batch_) {
        emit(items_[size_t(i)]);
        release(i);
      }
    }
  }

  void pend(uint32_t A, uint32_t B, cplx p) {
    Phase& P = pend_[A];
    P.used = true;
    used_ |= 1u << A;
    if (B == 0) { P.uniform *= p; return; }
    for (size_t i = 0; i < P.list.size(); ++i)
      if (P.list[i].mask == B) {
        P.list[i].p *= p;
        if (P.list[i].p == cplx(1.0, 0.0)) P.list.erase(P.list.begin() + long(i));
        return;
      }
    P.list.push_back(Entry{B, p});
  }

  // ---- emission -----------------------------------------------------------
  // Constant phases among the sets `which`: one table of all pending ones when
  // that is cheaper than one instruction each (per amplitude: 4 operations and
  // half a load in the table, 4 alone, 2 for a sign; 30 for an instruction).
  void join_constant(uint32_t which) {
    long alone = 0;
    for (uint32_t w = which; w; w &= w - 1) {
      const uint32_t A = uint32_t(ctz(w));
      const Phase& P = pend_[A];
      if (P.uniform == cplx(1.0, 0.0) || !P.list.empty()) continue;
      alone += 30 + (P.uniform == cplx(-1.0, 0.0) ? 2L : 4L) * long(kAll >> __builtin_popcount(A));
    }
    if (alone <= 30 + 9L * long(kAll) / 2) return;
    cplx v[32];
    for (cplx& x : v) x = cplx(1.0, 0.0);
    for (uint32_t w = used_; w; w &= w - 1) {
      const uint32_t A = uint32_t(ctz(w));
      const cplx u = pend_[A].uniform;
      if (u != cplx(1.0, 0.0))
        for (uint32_t r = A; r < kAll; r = (r + 1) | A) v[r] *= u;
      pend_[A].uniform = cplx(1.0, 0.0);
      if (pend_[A].list.empty()) drop(A);
    }
    // within half a turn of one another: shears around the middle, which goes to
    // the phase common to all amplitudes
    double d[64], lo = 0.0, hi = 0.0;
    const cplx first = std::conj(v[0]);
    if (!kF32) {
      for (uint32_t r = 0; r < kAll; ++r) {
        const cplx p = v[r] * first;
        d[r] = std::atan2(p.imag(), p.real());
        lo = std::min(lo, d[r]);
        hi = std::max(hi, d[r]);
      }
    } else if (!final_) {
      // the outermost by y / (|x| + |y|), which grows with the angle on each half turn
      cplx plo(1.0, 0.0), phi(1.0, 0.0);
      double olo = 0.0, ohi = 0.0;
      for (uint32_t r = 0; r < kAll; ++r) {
        const cplx p = v[r] * first;
        const double q = p.imag() / (std::fabs(p.real()) + std::fabs(p.imag()));
        const double o = p.real() >= 0.0 ? q : std::signbit(p.imag()) ? -2.0 - q : 2.0 - q;
        if (o < olo) olo = o, plo = p;
        if (o > ohi) ohi = o, phi = p;
      }
      lo = std::atan2(plo.imag(), plo.real());
      hi = std::atan2(phi.imag(), phi.real());
    }
    if (!final_ && hi - lo <= kHalfTurn) {
      const double mid = 0.5 * (lo + hi);
      const cplx m = v[0] * cplx(std::cos(mid), std::sin(mid));
      *global_ *= m;
      for (uint32_t r = kAll; r-- > 0;) {
        if (kF32) {  // tan(a / 2) = sin a / (1 + cos a) without an angle
          const cplx p = v[r] * std::conj(m);
          d[2 * r] = p.imag() / (1.0 + p.real());
          d[2 * r + 1] = p.imag();
        } else {
          const double a = d[r] - mid;
          d[2 * r] = std::tan(0.5 * a);
          d[2 * r + 1] = std::sin(a);
        }
      }
      W_.header(TC_TS, 0);
    } else {
      for (uint32_t r = 0; r < kAll; ++r) {
        d[2 * r] = v[r].real();
        d[2 * r + 1] = v[r].imag();
      }
      W_.header(TC_T, 0);
    }
    W_.reals(d, 2 * int(kAll));
    W_.end();
  }
  static constexpr double kHalfTurn = 3.14159265358979;
  void drop(uint32_t A) {
    pend_[A].clear();
    used_ &= ~(1u << A);
  }

  // Emit the pending phases that do not commute with a dense item on bits `t`.
  void flush(uint32_t t) {
    uint32_t which = 0;
    for (uint32_t w = used_ & ~1u; w; w &= w - 1)
      if (uint32_t(ctz(w)) & t) which |= w & (~w + 1);
    // the phase on all amplitudes can wait: it goes with the stage's last ones
    const cplx all = pend_[0].uniform;
    pend_[0].uniform = cplx(1.0, 0.0);
    join_constant(which);
    if (all != cplx(1.0, 0.0)) pend(0, 0, all);
    for (uint32_t w = which & used_; w; w &= w - 1) {
      put(uint32_t(ctz(w)), pend_[ctz(w)]);
      drop(uint32_t(ctz(w)));
    }
  }

  // Stage end: what is left; a list on all amplitudes joins one on a bit.
  void finish() {
    if (pend_[0].uniform != cplx(1.0, 0.0)) used_ |= 1u;
    join_constant(used_);
    const Phase& all = pend_[0];
    int join = -1;
    if (!all.trivial())
      for (int b = 0; b < kBits && join < 0; ++b) {
        const Phase& P = pend_[1u << b];
        if (P.used && !P.trivial() && !P.signs()) join = b;
      }
    for (uint32_t w = used_ & ~1u; w; w &= w - 1)
      if (join < 0 || ctz(w) != (1 << join)) put(uint32_t(ctz(w)), pend_[ctz(w)]);
    if (join < 0) put(0, all);
    else pair(join, all, pend_[1u << join]);
  }

  void put(uint32_t A, const Phase& P) {
    if (P.trivial()) return;
    const double u[2] = {P.uniform.real(), P.uniform.imag()};
    if (P.signs()) {
      if (P.list.empty()) {
        W_.header(TC_SG, A);
      } else {
        W_.header(TC_SL, A, uint32_t(P.list.size()));
        W_.head().w[2] = u[0] < 0 ? 1u : 0u;
        std::vector<uint32_t> v;
        for (const Entry& e : P.list) v.push_back(e.mask);
        W_.bytes(v.data(), v.size() * 4);
      }
    } else if (P.list.empty()) {
      const double ts[2] = {u[1] / (1.0 + u[0]), u[1]};
      const bool shear = kF32 && u[0] >= 0.0;
      W_.header(shear ? TC_PS : TC_PU, A);
      pair_of(shear ? ts : u);
    } else {
      W_.header(TC_PH, A, uint32_t(P.list.size()));
      if (kF32) W_.head().w[2] = turns(P.uniform);
      else W_.reals(u, 2);
      W_.list(P.list);
    }
    W_.end();
  }

  void pair(int b, const Phase& all, const Phase& bit) {
    W_.header(TC_D, uint32_t(b), uint32_t(all.list.size()) | uint32_t(bit.list.size()) << 16);
    if (kF32) {
      W_.head().w[2] = turns(all.uniform);
      W_.head().w[3] = turns(bit.uniform);
    } else {
      const double u[4] = {all.uniform.real(), all.uniform.imag(), bit.uniform.real(), bit.uniform.imag()};
      W_.reals(u, 4);
    }
    W_.list(all.list);
    W_.list(bit.list);
    W_.end();
  }

  // Two reals of an instruction: in the header (complex64) or the next word.
  void pair_of(const double* v) {
    if (kF32) {
      const float f[2] = {float(v[0]), float(v[1])};
      std::memcpy(&W_.head().w[2], f, 8);
    } else {
      W_.reals(v, 2);
    }
  }

  // The rotations of a batch (distinct bits) as one instruction.
  void emit_rotations(Item::Kind kind) {
    uint32_t bits = 0;
    double v[5][2] = {};
    for (int i : batch_) {
      const Item& I = items_[size_t(i)];
      if (I.kind != kind) continue;
      bits |= I.dense;
      v[ctz(I.dense)][0] = I.t;
      v[ctz(I.dense)][1] = I.s;
    }
    if (!bits) return;
    W_.header(kind == Item::ROT ? TC_R : TC_X, 0, bits);
    if (kF32) pair_of(v[0]);
    W_.reals(kF32 ? v[1] : v[0], kF32 ? 2 * (kBits - 1) : 2 * kBits);
    W_.end();
  }

  void emit(const Item& I) {
    if (I.kind == Item::GENERIC) {
      double v[8];
      for (int i = 0; i < 4; ++i) { v[2 * i] = I.m[i].real(); v[2 * i + 1] = I.m[i].imag(); }
      W_.header(TC_G, uint32_t(ctz(I.dense)), I.cnr);
      W_.reals(v, 8);
      W_.end();
    } else if (I.kind == Item::FLIP) {
      W_.header(TC_OP, OP_X1, uint32_t(ctz(I.dense)));
      W_.end();
    } else if (I.kind == Item::RECORD) {
      const TileOp<Real>& t = enc_[I.op];
      if (t.kind == OP_U1 && (t.creg & (t.creg - 1))) {
        // the kernel's 2x2 takes one register control: the first of several becomes
        // the second bit of a 4x4 that is the identity where it is 0
        const uint32_t c = uint32_t(ctz(t.creg));
        W_.header(TC_OP, OP_U2, uint32_t(t.rb0) | c << 8 | (t.creg & (t.creg - 1u)) << 16);
        W_.head().w[2] = t.cnr;
        Real m[32] = {};
        m[0] = m[2 * 5] = Real(1);
        for (int r = 0; r < 2; ++r)
          for (int e = 0; e < 4; ++e) m[2 * (4 * (2 + r) + 2) + e] = t.m[4 * r + e];
        W_.bytes(m, sizeof(m));
        W_.end();
        return;
      }
      W_.header(TC_OP, t.kind, uint32_t(t.rb0) | uint32_t(t.rb1) << 8 | uint32_t(t.creg) << 16);
      W_.head().w[2] = t.cnr;
      const size_t entries = t.kind == OP_U2 ? 16 : t.kind == OP_U1 ? 4 : 0;
      W_.bytes(t.m, 2 * sizeof(Real) * entries);
      W_.end();
    }
  }

  static int ctz(uint32_t v) { return __builtin_ctz(v); }

  const std::vector<Op>& ops_;
  const TilePlan& plan_;
  const std::vector<TileOp<Real>>& enc_;
  Writer W_;
  std::vector<Item> items_;
  uint32_t dense_bits_ = 0;  // register bits some item changes
  struct Edge {
    int to, next;
  };
  std::vector<int> wait_, first_;  // per item: items it waits for; its first edge
  std::vector<Edge> edges_;
  std::vector<int> phases_, dense_, batch_;  // items that wait for nothing; those being emitted
  std::vector<int> readers_[kBits];
  Phase pend_[32];
  uint32_t used_ = 0;  // pend_ entries in use
  cplx* global_ = nullptr;  // phase common to all amplitudes
  bool final_ = false;      // emitting the plan's last phases: nothing takes a common one any more
  cplx acc_[5][4];
  bool have_[5];
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
  t[StageTab::UL] = t[StageTab::UH] = t[StageTab::SL] = t[StageTab::SH] = 0;
  for (int j = 0; j < 4; ++j) {  // each bit on top of the combinations of those below it
    const uint32_t lo = j < S.n_tbits ? 1u << S.tpos[j] : 0u, hi = j + 4 < S.n_tbits ? 1u << S.tpos[j + 4] : 0u;
    const uint32_t slo = swz(lo), shi = swz(hi);
    for (int v = 0; v < 1 << j; ++v) {
      const int w = v | 1 << j;
      t[StageTab::UL + w] = t[StageTab::UL + v] | lo;
      t[StageTab::UH + w] = t[StageTab::UH + v] | hi;
      t[StageTab::SL + w] = t[StageTab::SL + v] ^ slo;
      t[StageTab::SH + w] = t[StageTab::SH + v] ^ shi;
    }
  }
}

template <typename Real>
void compile(const std::vector<Op>& ops, TilePlan* plan, const std::vector<TileOp<Real>>& enc) {
  StageCompiler<Real> C(ops, *plan, enc);
  cplx global(1.0, 0.0);
  const size_t last = plan->stages.empty() ? 0 : plan->stages.size() - 1;
  // the tables, and about what an op's share of the instructions takes
  plan->prog.reserve(plan->stages.size() * (kStageTabWords / 4 + 8) + 2 * plan->op_src.size() + 64);
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

// A unitary 2x2 without controls that is not real, diagonal or anti-diagonal: its
// three Euler angles are all there.  `rx`: of RX's form.
bool takes_carry(const Op& o, bool* rx) {
  if (o.kind != OP_U1 || o.nctrl != 0) return false;
  const cplx* m = o.m;
  const double eps = 1e-12;
  if (std::abs(std::norm(m[0]) + std::norm(m[2]) - 1.0) > eps || std::abs(std::norm(m[1]) + std::norm(m[3]) - 1.0) > eps ||
      std::norm(std::conj(m[0]) * m[1] + std::conj(m[2]) * m[3]) > eps * eps)
    return false;
  const bool real = m[0].imag() == 0 && m[1].imag() == 0 && m[2].imag() == 0 && m[3].imag() == 0;
  *rx = m[0].imag() == 0 && m[1].real() == 0 && m[2].real() == 0 && m[3].imag() == 0;
  return !real && std::norm(m[0]) > 1e-12 && std::norm(m[2]) > 1e-12;
}

void times(const cplx* a, const cplx* b, cplx* out) {
  const cplx r[4] = {a[0] * b[0] + a[1] * b[2], a[0] * b[1] + a[1] * b[3], a[2] * b[0] + a[3] * b[2],
                     a[2] * b[1] + a[3] * b[3]};
  std::memcpy(static_cast<void*>(out), r, sizeof(r));
}

}  // namespace

std::vector<Op> carry_phases(std::vector<Op> ops) {
  size_t takers = 0;
  struct Takes {
    bool any, rx;
  };
  std::vector<Takes> takes(ops.size());
  for (size_t i = 0; i < ops.size(); ++i) takers += takes[i].any = takes_carry(ops[i], &takes[i].rx);
  if (takers < 2) return ops;
  // the op after op i on each of its (at most five) qubits, from a backward walk
  struct Next {
    int8_t q[5];
    int32_t op[5];
    int n = 0;
  };
  std::vector<Next> next(ops.size());
  int32_t seen[64];
  for (int32_t& v : seen) v = -1;
  for (size_t i = ops.size(); i-- > 0;)
    for (uint64_t m = ops[i].qubit_mask(); m; m &= m - 1) {
      const int q = __builtin_ctzll(m);
      next[i].q[next[i].n] = int8_t(q);
      next[i].op[next[i].n++] = seen[q];
      seen[q] = int32_t(i);
    }
  auto after = [&](size_t i, int q) {
    for (int k = 0; k < next[i].n; ++k)
      if (next[i].q[k] == q) return next[i].op[k];
    return -1;
  };
  for (size_t i = 0; i < ops.size(); ++i) {
    if (!takes[i].any) continue;
    const bool rx = takes[i].rx;
    const int q = ops[i].t0;
    bool z = true, x = true, found = false;
    size_t e = 0;
    for (int32_t k = after(i, q); k >= 0 && (z || x); k = after(size_t(k), q)) {
      const Op& o = ops[size_t(k)];
      if (takes[size_t(k)].any) {
        e = size_t(k);
        found = true;
        break;
      }
      if (o.diagonal() || ((o.ctrl_mask() >> q) & 1)) x = false;
      else if (o.kind == OP_X1 && o.t0 == q) z = false;
      else z = x = false;
    }
    // none, nothing between (the compiler merges the two), or an RX that would
    // wander whole through X targets
    if (!found || z == x || (rx && x)) continue;
    cplx* m = ops[i].m;
    cplx w[4] = {m[0], m[1], m[2], m[3]}, c[4] = {1.0, 0.0, 0.0, 1.0};
    if (z) {
      const cplx p = (m[2] / std::abs(m[2])) / (m[0] / std::abs(m[0]));
      c[3] = p;
      w[2] = m[2] / p;
      w[3] = m[3] / p;
    } else {
      // RX(al) rotation phase: RX(-al) m has a real ratio in its first column
      const double al = std::atan2(-2.0 * (std::conj(m[0]) * m[2]).imag(), std::norm(m[0]) - std::norm(m[2]));
      const double ch = std::cos(al / 2), sh = std::sin(al / 2);
      const cplx rx[4] = {ch, cplx(0, -sh), cplx(0, -sh), ch}, inv[4] = {ch, cplx(0, sh), cplx(0, sh), ch};
      std::memcpy(static_cast<void*>(c), rx, sizeof(c));
      times(inv, m, w);
    }
    std::memcpy(static_cast<void*>(m), w, sizeof(w));
    times(ops[e].m, c, ops[e].m);
    takes[e].any = takes_carry(ops[e], &takes[e].rx);
  }
  return ops;
}

void build_tile_prog(const std::vector<Op>& ops, TilePlan* plan) {
  plan->prog.clear();
  if (plan->dt == DType::C64) compile<float>(ops, plan, plan->ops_f);
  else compile<double>(ops, plan, plan->ops_d);
  plan->stats.upload_bytes = plan->passes.size() * sizeof(PassRec) + plan->prog.size() * sizeof(ProgWord);
}

}  // namespace nqpu
