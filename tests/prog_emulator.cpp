// Test infrastructure: an interpreter of the tiled passes' stage programs
// (nqpu_b200/csrc/tileprog.h) on the CPU, in FP64 over the encoded operands.  It
// walks the state block by block (the amplitudes that differ in a stage's
// register bits), runs the stage's words and applies the write-back permutation.
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <vector>

#include "planner.h"
#include "tileprog.h"

using namespace nqpu;
using cd = std::complex<double>;

namespace {

template <typename Real>
cd cget(const ProgWord* q, int i) {
  Real v[2];
  std::memcpy(v, reinterpret_cast<const char*>(q) + size_t(i) * 2 * sizeof(Real), sizeof(v));
  return cd(double(v[0]), double(v[1]));
}
cd turn(uint32_t a) {
  const double t = 6.283185307179586476925 * (double(a) / 4294967296.0);
  return cd(std::cos(t), std::sin(t));
}

void record(const TileOp<float>* f, const TileOp<double>* d, std::vector<cd>& a, uint32_t vbase) {
  auto m = [&](int i) { return f ? cd(f->m[2 * i], f->m[2 * i + 1]) : cd(d->m[2 * i], d->m[2 * i + 1]); };
  const uint8_t kind = f ? f->kind : d->kind;
  const uint32_t t0 = 1u << (f ? f->rb0 : d->rb0), t1 = 1u << (f ? f->rb1 : d->rb1), creg = f ? f->creg : d->creg;
  const uint32_t cnr = f ? f->cnr : d->cnr;
  if ((vbase & cnr) != cnr) return;
  for (uint32_t i = 0; i < a.size(); ++i) {
    if ((i & creg) != creg || (i & t0)) continue;
    const cd x = a[i], y = a[i | t0];
    if (kind == OP_U1) { a[i] = m(0) * x + m(1) * y; a[i | t0] = m(2) * x + m(3) * y; }
    if (kind == OP_X1) std::swap(a[i], a[i | t0]);
    if ((kind == OP_U2 || kind == OP_SW) && (i & t1)) continue;
    if (kind == OP_SW) std::swap(a[i | t0], a[i | t1]);
    if (kind == OP_U2) {
      const uint32_t ix[4] = {i, i | t0, i | t1, i | t0 | t1};
      cd v[4];
      for (int r = 0; r < 4; ++r) {
        v[r] = 0;
        for (int c = 0; c < 4; ++c) v[r] += m(4 * r + c) * a[ix[c]];
      }
      for (int r = 0; r < 4; ++r) a[ix[r]] = v[r];
    }
  }
}

template <typename Real>
int run_words(const ProgWord* p, const ProgWord* end, std::vector<cd>& a, uint32_t vbase) {
  constexpr bool F32 = sizeof(Real) == 4;
  auto hit = [&](uint32_t m) { return (vbase & m) == m; };
  auto list = [&](const ProgWord*& q, uint32_t n, cd v) {
    for (uint32_t i = 0; i < n; ++i) {
      if (F32) {
        if (hit(q[i / 2].w[2 * (i & 1)])) v *= turn(q[i / 2].w[2 * (i & 1) + 1]);
      } else if (hit(q[2 * i].w[0])) {
        v *= cget<double>(q + 2 * i + 1, 0);
      }
    }
    q += F32 ? (n + 1) / 2 : 2 * n;
    return v;
  };
  while (p < end) {
    const uint32_t code = p->w[0] & 0xFFu, arg = (p->w[0] >> 8) & 0xFFu, len = p->w[0] >> 16;
    const ProgWord* q = p + 1;
    const ProgWord& h = *p;
    if (len == 0 || p + len > end) return -2;
    const cd two = F32 ? cget<float>(p, 1) : cget<double>(q, 0);  // the instruction's two reals
    auto turn_by = [](bool shear, cd p, cd& v) {
      if (!shear) { v *= p; return; }
      double x = v.real() - p.real() * v.imag();
      const double y = v.imag() + p.imag() * x;
      x -= p.real() * y;
      v = cd(x, y);
    };
    auto two_by_two = [&](uint32_t b, const cd* m) {
      for (uint32_t i = 0; i < a.size(); ++i) {
        if (i & b) continue;
        const cd x = a[i], y = a[i | b];
        a[i] = m[0] * x + m[1] * y;
        a[i | b] = m[2] * x + m[3] * y;
      }
    };
    if (code == TC_R || code == TC_X) {
      if (h.w[1] >= a.size()) return -3;
      for (int b = 0; (1u << b) < a.size(); ++b) {
        if (!((h.w[1] >> b) & 1)) continue;
        // the three shears as one matrix
        const cd ts = F32 ? (b ? cget<float>(q, b - 1) : two) : cget<double>(q, b);
        const double t = ts.real(), s = ts.imag(), c = 1 - t * s, o = t * (2 - t * s);
        const cd f = code == TC_X ? cd(0, 1) : cd(1, 0);
        const cd m[4] = {c, -f * o, (code == TC_X ? -f : f) * s, c};
        two_by_two(1u << b, m);
      }
    } else if (code == TC_G) {
      cd m[4];
      for (int i = 0; i < 4; ++i) m[i] = cget<Real>(q, i);
      if (hit(h.w[1])) two_by_two(1u << arg, m);
    } else if (code == TC_T || code == TC_TS) {
      for (uint32_t i = 0; i < a.size(); ++i) turn_by(code == TC_TS, cget<Real>(q, int(i)), a[i]);
    } else if (code == TC_PU || code == TC_PS) {
      for (uint32_t i = 0; i < a.size(); ++i)
        if ((i & arg) == arg) turn_by(code == TC_PS, two, a[i]);
    } else if (code == TC_SG || code == TC_SL) {
      uint32_t s = code == TC_SG ? 1u : h.w[2];
      for (uint32_t i = 0; code == TC_SL && i < h.w[1]; ++i) s += hit(q[i / 4].w[i & 3]);
      for (uint32_t i = 0; i < a.size(); ++i)
        if ((i & arg) == arg && (s & 1)) a[i] = -a[i];
    } else if (code == TC_PH) {
      if (!F32) ++q;
      const cd v = list(q, h.w[1], F32 ? turn(h.w[2]) : two);
      for (uint32_t i = 0; i < a.size(); ++i)
        if ((i & arg) == arg) a[i] *= v;
    } else if (code == TC_D) {
      const uint32_t b = 1u << arg;
      cd d0 = F32 ? turn(h.w[2]) : two, d1 = F32 ? turn(h.w[3]) : cget<double>(q, 1);
      if (!F32) q += 2;
      d0 = list(q, h.w[1] & 0xFFFFu, d0);
      d1 = d0 * list(q, h.w[1] >> 16, d1);
      for (uint32_t i = 0; i < a.size(); ++i) a[i] *= (i & b) ? d1 : d0;
    } else {
      TileOp<Real> t;
      t.kind = uint8_t(arg);
      t.rb0 = uint8_t(h.w[1]);
      t.rb1 = uint8_t(h.w[1] >> 8);
      t.creg = uint8_t(h.w[1] >> 16);
      t.cnr = h.w[2];
      if (size_t(len) * 16 != 16 + 2 * sizeof(Real) * (arg == OP_U2 ? 16 : arg == OP_U1 ? 4 : 0)) return -5;
      std::memcpy(t.m, q, size_t(len - 1) * 16);
      record(F32 ? reinterpret_cast<TileOp<float>*>(&t) : nullptr, F32 ? nullptr : reinterpret_cast<TileOp<double>*>(&t),
             a, vbase);
    }
    p += len;
  }
  return p == end ? 0 : -4;
}

uint32_t swz(uint32_t u) {
  uint32_t f = 0;
  for (uint32_t w = u >> 3; w; w >>= 3) f ^= w & 7u;
  return u ^ f;
}

// The stage table addresses every slot of the tile once on the way in and once on
// the way out, at the places the stage record names.
int check_tab(const PassRec& P, const StageRec& S, int vb, const uint32_t* T) {
  if (T[StageTab::OB] != uint32_t(S.prog_begin) || T[StageTab::OE] != uint32_t(S.prog_end)) return 1;
  const uint32_t nvec = 1u << (P.k - vb);
  const int nrb = vb + kRegFree;
  std::vector<int> in(size_t(nvec), 0), outs(size_t(nvec) << vb, 0);
  for (uint32_t tid = 0; tid < nvec / 16; ++tid) {
    uint32_t u = 0;
    for (int j = 0; j < S.n_tbits; ++j) u |= ((tid >> j) & 1u) << S.tpos[j];
    const uint32_t ub = T[StageTab::UL + (tid & 15)] | T[StageTab::UH + (tid >> 4)];
    const uint32_t sb = T[StageTab::SL + (tid & 15)] ^ T[StageTab::SH + (tid >> 4)];
    if (ub != u || sb != swz(u)) return 2;
    for (uint32_t r = 0; r < 16; ++r) {
      uint32_t v = u, slot = sb;
      for (int i = 0; i < 4; ++i)
        if ((r >> i) & 1) { v |= 1u << (S.rpos[i] - vb); slot ^= T[StageTab::S + i]; }
      if (slot != swz(v) || slot >= nvec || in[slot]++) return 3;
    }
    // one combination of the conditional translations per thread
    uint32_t w = uint32_t(S.sbx), ws = T[StageTab::WS], wh = T[StageTab::WH];
    if (T[StageTab::NC] != uint32_t(S.ncond)) return 4;
    for (int i = 0; i < S.ncond; ++i) {
      if (T[StageTab::CC + i] != S.cond_cnr[i]) return 5;
      if ((tid >> i) & 1) { w ^= uint32_t(S.cond_w[i]); ws ^= T[StageTab::CS + i]; wh ^= T[StageTab::CH + i]; }
    }
    for (uint32_t p = 0; p < (1u << nrb); ++p) {
      uint32_t m = w, slot = sb ^ ws, h = wh;
      for (int j = 0; j < nrb; ++j)
        if ((p >> j) & 1) m ^= uint32_t(S.scol[j]);
      for (int i = 0; i < 4; ++i)
        if ((p >> (vb + i)) & 1) { slot ^= T[StageTab::CW + i]; h ^= (T[StageTab::HB] >> i) & 1; }
      if (vb && (p & 1)) { slot ^= T[StageTab::CZ]; h ^= T[StageTab::HZ]; }
      uint32_t v = u;
      for (int i = 0; i < 4; ++i)
        if ((m >> (vb + i)) & 1) v |= 1u << (S.rpos[i] - vb);
      if (slot != swz(v) || (vb && h != (m & 1)) || outs[(size_t(slot) << vb) | (vb ? h : 0)]++) return 6;
    }
  }
  return vb && T[StageTab::MZ] != uint32_t(S.scol[0]) ? 7 : 0;
}

}  // namespace

// Run the compiled plan on `state`; stats[0..2] = ops the plan encodes, program
// instructions (all passes), passes.
extern "C" int prog_run(int n, int c64, int kmax, const double* flat, int ngates, double* state, int64_t* stats) {
  std::vector<GateRec> gates(ngates);
  for (int i = 0; i < ngates; ++i) {
    const double* g = flat + size_t(i) * 40;
    GateRec& r = gates[i];
    r.code = uint8_t(g[0]);
    r.nq = uint8_t(gate_arity(r.code));
    for (int j = 0; j < 3; ++j) r.q[j] = int(g[1 + j]);
    for (int j = 0; j < 4; ++j) r.p[j] = g[4 + j];
    for (int j = 0; j < 16; ++j) r.m[j] = cplx(g[8 + 2 * j], g[9 + 2 * j]);
  }
  const DType dt = c64 ? DType::C64 : DType::C128;
  const int vb = c64 ? 1 : 0, nrb = vb + kRegFree;
  TilePlan plan;
  std::string err;
  const std::vector<Op> ops = carry_phases(lower_circuit(gates));
  if (!build_tile_plan(ops, n, dt, kmax, &plan, &err)) return -1;
  build_tile_prog(ops, &plan);
  stats[0] = int64_t(plan.op_src.size());
  stats[1] = 0;
  stats[2] = int64_t(plan.passes.size());
  const size_t dim = size_t(1) << n;
  std::vector<cd> st(dim), next(dim);
  for (size_t i = 0; i < dim; ++i) st[i] = cd(state[2 * i], state[2 * i + 1]);
  for (const PassRec& P : plan.passes) {
    const size_t tw = size_t(P.stage_end - P.stage_begin) * (kStageTabWords / 4);
    for (size_t i = tw; i + 1 < size_t(P.prog_words); i += plan.prog[size_t(P.prog_begin) + i].w[0] >> 16) ++stats[1];
    auto qubit = [&](int tb) { return tb < P.c ? tb : P.qhi[tb - P.c]; };
    for (int s = P.stage_begin; s < P.stage_end; ++s) {
      const StageRec& S = plan.stages[size_t(s)];
      uint64_t rq[5], regs = 0;
      for (int j = 0; j < nrb; ++j) {
        rq[j] = 1ull << ((vb && j == 0) ? 0 : qubit(S.rpos[j - vb]));
        regs |= rq[j];
      }
      if (S.prog_begin < 0 || S.prog_end + int(tw) > P.prog_words) return -5;
      uint32_t T[kStageTabWords];
      std::memcpy(T, plan.prog.data() + P.prog_begin + size_t(s - P.stage_begin) * (kStageTabWords / 4), sizeof(T));
      if (check_tab(P, S, vb, T)) return -6;
      for (uint64_t base = 0; base < dim; ++base) {
        if (base & regs) continue;
        uint32_t vbase = 0;
        for (int tb = 0; tb < P.k; ++tb) vbase |= uint32_t((base >> qubit(tb)) & 1) << tb;
        for (int j = 0; j < P.n_ext; ++j) vbase |= uint32_t((base >> P.ext[j]) & 1) << (P.k + j);
        auto at = [&](uint32_t m) {
          uint64_t i = base;
          for (int j = 0; j < nrb; ++j)
            if ((m >> j) & 1) i |= rq[j];
          return i;
        };
        std::vector<cd> a(size_t(1) << nrb);
        for (uint32_t p = 0; p < a.size(); ++p) a[p] = st[at(p)];
        const ProgWord* w = plan.prog.data() + P.prog_begin + (P.stage_end - P.stage_begin) * (kStageTabWords / 4);
        const int rc = c64 ? run_words<float>(w + S.prog_begin, w + S.prog_end, a, vbase)
                           : run_words<double>(w + S.prog_begin, w + S.prog_end, a, vbase);
        if (rc) return rc;
        uint32_t x = uint32_t(S.sbx);
        for (int i = 0; i < S.ncond; ++i)
          if ((vbase & S.cond_cnr[i]) == S.cond_cnr[i]) x ^= uint32_t(S.cond_w[i]);
        for (uint32_t p = 0; p < a.size(); ++p) {
          uint32_t m = x;
          for (int j = 0; j < nrb; ++j)
            if ((p >> j) & 1) m ^= uint32_t(S.scol[j]);
          next[at(m)] = a[p];
        }
      }
      st.swap(next);
    }
  }
  for (size_t i = 0; i < dim; ++i) { state[2 * i] = st[i].real(); state[2 * i + 1] = st[i].imag(); }
  return 0;
}
