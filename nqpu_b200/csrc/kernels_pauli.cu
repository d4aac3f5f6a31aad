// Pauli sums: sum_t c_t <P_t> of many Pauli strings in one launch
// (expectation_pauli_string / expectation of a Hamiltonian, R/lib.rs:465,518).
//
// With coeff(i) = i^ny (-1)^popcount(i & z), a string contributes
// sum_i Re(conj(a_i) coeff(i) a_{i ^ x}).  For x = 0 that is |a_i|^2 with a
// sign; for x != 0 the amplitudes i and i ^ x contribute the same value, so one
// term per pair is enough: 2 (-1)^{ny/2} (-1)^{pc(i & z)} Re(conj(a_i) a_{i^x})
// for an even number of Y's and -+2 (...) Im(...) for an odd one.
//
// The host groups the strings into register sets of four qubits (pauli_plan): a
// thread loads the 16 amplitudes that differ in a set's qubits, converts them to
// FP64 once, and evaluates every string whose X|Y positions lie inside the set on
// them.  Diagonal strings take a Walsh-Hadamard transform of the 16
// probabilities: the sum of |a|^2 over the block with any sign pattern on its
// four qubits is one of its 16 outputs, so a string costs one sign and one
// addition per 16 amplitudes.
//
// Bound: an n-qubit Ising Hamiltonian takes ceil(n / 4) sets, each a read of the
// state.  The sets whose qubits lie below kPauliChunkBits run chunk by chunk, so
// all but the first of them find the chunk in L2.  FP64 conversion (two per
// complex64 amplitude and set) comes second.  Before, each string was a launch
// of its own that read the state with 4-byte loads (and its partner amplitudes
// again) and ended in a host synchronisation.  Measured: the 24-qubit Ising
// Hamiltonian (47 strings, complex64) 3140 -> 190 us.
#include "reduce_device.cuh"

namespace nqpu {

// 2^22 amplitudes are 32 MB (complex64) / 64 MB (complex128): well inside the L2.
constexpr int kPauliChunkBits = 22;

// Complex128 from this size on (128 MB of state): a set that holds qubits 0, 1 and 2
// reads 128 bytes per lane, a line each, and for one string alone the scalar kernel
// is the faster one (25 qubits, X on 0, 1, 2: 108 us, 154 from a set; on 3, 4, 5: 104).
constexpr int kPauliAloneQubits = 23;

void pauli_plan(DType dt, const PauliString* strings, size_t count, int n, PauliPlan* plan,
                std::vector<PauliString>* wide) {
  plan->sets.clear();
  plan->terms.clear();
  wide->clear();
  struct Group {
    uint64_t bits = 0;
    std::vector<size_t> idx;
  };
  std::vector<Group> groups;
  std::vector<size_t> diag;
  for (size_t t = 0; t < count; ++t) {
    const uint64_t x = strings[t].x;
    if (x == 0) { diag.push_back(t); continue; }
    if (__builtin_popcountll(x) > 4) { wide->push_back(strings[t]); continue; }
    Group* g = nullptr;
    for (Group& h : groups)
      if (__builtin_popcountll(h.bits | x) <= 4) { g = &h; break; }
    if (!g) { groups.emplace_back(); g = &groups.back(); }
    g->bits |= x;
    g->idx.push_back(t);
  }
  if (dt == DType::C128 && n >= kPauliAloneQubits)
    for (size_t i = groups.size(); i-- > 0;)
      if (groups[i].idx.size() == 1 && (groups[i].bits & 7) == 7) {
        wide->push_back(strings[groups[i].idx[0]]);
        groups.erase(groups.begin() + long(i));
      }
  if (!diag.empty()) {
    if (groups.empty()) groups.emplace_back();
    groups[0].idx.insert(groups[0].idx.end(), diag.begin(), diag.end());
  }
  // fill every set to four qubits, highest first (a set without low qubits loads
  // whole lines per warp)
  for (Group& g : groups)
    for (int q = std::min(n, kPauliChunkBits) - 1; q >= 0 && __builtin_popcountll(g.bits) < 4; --q) g.bits |= 1ull << q;
  std::stable_sort(groups.begin(), groups.end(), [](const Group& a, const Group& b) {
    return (a.bits >> kPauliChunkBits != 0) < (b.bits >> kPauliChunkBits != 0);
  });
  for (const Group& g : groups) {
    PauliSet S{};
    int nb = 0;
    for (int q = 0; q < n; ++q)
      if ((g.bits >> q) & 1) S.rbit[nb++] = uint8_t(q);
    auto inside = [&](uint64_t m) {
      int v = 0;
      for (int b = 0; b < 4; ++b) v |= int((m >> S.rbit[b]) & 1) << b;
      return v;
    };
    // (X positions, Z positions) within the set order the terms
    std::vector<std::pair<int, size_t>> order;
    for (size_t t : g.idx) {
      const PauliString& P = strings[t];
      if (P.z == 0 && P.x != 0 && (P.x & (P.x - 1)) == 0) {
        const int b = __builtin_ctz(unsigned(inside(P.x)));
        S.plain |= uint16_t(1u << b);
        S.cx[b] += 2.0 * P.c;
        continue;
      }
      order.push_back({inside(P.x) * 16 + inside(P.z), t});
    }
    std::stable_sort(order.begin(), order.end(),
                     [](const std::pair<int, size_t>& a, const std::pair<int, size_t>& b) { return a.first < b.first; });
    size_t k = 0;
    for (int m = 0; m <= 16; ++m) {
      while (k < order.size() && order[k].first < 16 * m) ++k;
      S.beg[m] = uint16_t(plan->terms.size() + k);
      if (m > 0 && S.beg[m] > S.beg[m - 1] && m - 1 > 0) S.xused |= uint16_t(1u << (m - 1));
    }
    k = 0;
    for (int m = 0; m <= 16; ++m) {
      while (k < order.size() && order[k].first < m) ++k;
      S.dbeg[m] = uint16_t(plan->terms.size() + k);
      if (m > 0 && S.dbeg[m] > S.dbeg[m - 1]) S.dused |= uint16_t(1u << (m - 1));
    }
    for (const auto& o : order) {
      const PauliString& P = strings[o.second];
      const int ny = __builtin_popcountll(P.y) & 3;
      PauliTerm T;
      T.z = (P.z & ~g.bits) | (uint64_t(inside(P.z)) << 60) | (uint64_t(ny & 1) << 59);
      T.c = P.x == 0 ? P.c : 2.0 * P.c * ((ny == 1 || ny == 2) ? -1.0 : 1.0);
      plan->terms.push_back(T);
    }
    plan->sets.push_back(S);
  }
}

__device__ __forceinline__ double flip(double v, uint32_t bit) {  // -v when bit 0 of `bit` is set
  return __hiloint2double(__double2hiint(v) ^ int(bit << 31), __double2loint(v));
}

template <typename Real>
__global__ void __launch_bounds__(kRedThreads, 2)
    k_pauli_sum(const Real* __restrict__ amp, int n, const PauliSet* __restrict__ sets, int nlow, int nsets,
                const PauliTerm* __restrict__ terms, double* __restrict__ part, double* __restrict__ out) {
  using C = typename Tr<Real>::C;
  const C* a = reinterpret_cast<const C*>(amp);
  const int hbits = n < kPauliChunkBits ? n : kPauliChunkBits;
  // work units of kRedThreads threads, one block after the other: first (chunk,
  // low set, tile) with the tile running fastest, then (high set, tile).  The
  // counters step instead of dividing the unit number (a 64-bit division costs
  // as much as a whole unit's arithmetic).
  const uint32_t low_tiles = 1u << max(0, hbits - 12), high_tiles = 1u << max(0, n - 12);
  uint32_t tile = blockIdx.x, chunk = 0;
  int si = 0;
  KSum acc;
  for (;; tile += gridDim.x) {
    while (si < nlow && tile >= low_tiles) {
      tile -= low_tiles;
      if (++si == nlow && ++chunk < (1u << (n - hbits))) si = 0;
    }
    while (si >= nlow && si < nsets && tile >= high_tiles) {
      tile -= high_tiles;
      ++si;
    }
    if (si >= nsets) break;
    const bool low = si < nlow;
    const uint32_t w = tile * kRedThreads + threadIdx.x;
    if (w >> ((low ? hbits : n) - 4)) continue;  // fewer work items than threads
    const PauliSet* S = sets + si;
    uint64_t base = w, off[4];
    const uint32_t rb = *reinterpret_cast<const uint32_t*>(S->rbit);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int q = int((rb >> (8 * b)) & 0xFF);
      off[b] = 1ull << q;
      const uint64_t lo = base & (off[b] - 1);
      base += base - lo;  // insert a zero bit at q
    }
    if (low) base += uint64_t(chunk) << hbits;
    C v[16];
    const C* p4[4];  // the four combinations of the upper two bits
    p4[0] = a + base;
    p4[1] = p4[0] + off[2];
    p4[2] = p4[0] + off[3];
    p4[3] = p4[1] + off[3];
    const uint64_t off01 = off[0] + off[1];
    auto at = [&](int r) { return p4[r >> 2] + ((r & 3) == 0 ? 0 : (r & 3) == 1 ? off[0] : (r & 3) == 2 ? off[1] : off01); };
    if (sizeof(Real) == 4 && off[0] == 1) {  // qubit 0 in the set: pairs as 128-bit loads
#pragma unroll
      for (int r = 0; r < 16; r += 2) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(at(r)));
        v[r].x = x.x; v[r].y = x.y; v[r + 1].x = x.z; v[r + 1].y = x.w;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = __ldg(at(r));
    }
    double re[16], im[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      re[r] = v[r].x;
      im[r] = v[r].y;
    }
    double item = 0.0;
    auto term = [&](int t, double* c) {
      const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(terms + t));
      *c = __longlong_as_double((long long)x.y);
      return x.x;
    };
    constexpr uint64_t kOutside = (1ull << 59) - 1;
    const uint32_t dused = S->dused, xused = S->xused;
    if (dused) {
      double W[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) W[r] = re[r] * re[r] + im[r] * im[r];
#pragma unroll
      for (int b = 1; b < 16; b <<= 1)
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (!(r & b)) {
            const double x = W[r], y = W[r | b];
            W[r] = x + y;
            W[r | b] = x - y;
          }
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        if (!((dused >> m) & 1)) continue;
        const int e = S->dbeg[m + 1];
        double cs = 0.0;
        for (int t = S->dbeg[m]; t < e; ++t) {
          double c;
          const uint64_t z = term(t, &c);
          cs += flip(c, uint32_t(__popcll(base & z & kOutside)));
        }
        item += W[m] * cs;
      }
    }
    // a single X: no sign anywhere
    const uint32_t plain = S->plain;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (!((plain >> b) & 1)) continue;
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (!(r & (1 << b))) {
          s0 = fma(re[r], re[r | (1 << b)], s0);
          s1 = fma(im[r], im[r | (1 << b)], s1);
        }
      item = fma(S->cx[b], s0 + s1, item);
    }
    if (xused)
#pragma unroll
    for (int m = 1; m < 16; ++m) {
      if (!((xused >> m) & 1)) continue;
      const int top = m >= 8 ? 8 : m >= 4 ? 4 : m >= 2 ? 2 : 1;
      const int e = S->beg[m + 1];
      for (int t = S->beg[m]; t < e; ++t) {
        double c;
        const uint64_t z = term(t, &c);
        const uint32_t zr = uint32_t(z >> 60);
        // bit r: parity of r & zr
        const uint32_t pat = ((zr & 1) ? 0xAAAAu : 0u) ^ ((zr & 2) ? 0xCCCCu : 0u) ^ ((zr & 4) ? 0xF0F0u : 0u) ^
                             ((zr & 8) ? 0xFF00u : 0u);
        double s = 0.0;
        if ((z >> 59) & 1) {
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (!(r & top)) s += flip(re[r] * im[r ^ m] - im[r] * re[r ^ m], pat >> r);
        } else if (zr == 0) {
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (!(r & top)) s += re[r] * re[r ^ m] + im[r] * im[r ^ m];
        } else {
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (!(r & top)) s += flip(re[r] * re[r ^ m] + im[r] * im[r ^ m], pat >> r);
        }
        item += flip(c * s, uint32_t(__popcll(base & z & kOutside)));
      }
    }
    acc.add(item);
  }
  __shared__ double sh[kRedWarps];
  const double r = warp_sum(acc.s);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kRedWarps; ++w) t += sh[w];
    if (gridDim.x == 1) out[0] = t;
    else part[blockIdx.x] = t;
  }
}

cudaError_t launch_pauli_sum(DType dt, const void* amp, int n, const PauliSet* d_sets, const PauliPlan& plan,
                             const PauliTerm* d_terms, double* scratch, double* out, cudaStream_t s, int num_sms) {
  int nlow = 0;
  for (const PauliSet& S : plan.sets) nlow += S.rbit[3] < kPauliChunkBits;
  const int nsets = int(plan.sets.size());
  const uint64_t units = (uint64_t(nsets) << n) >> 12;  // of 256 threads x 16 amplitudes
  const unsigned g = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(std::max<uint64_t>(units, uint64_t(nsets)),
                                                                       uint64_t(num_sms) * 2)));
  if (dt == DType::C64)
    k_pauli_sum<float><<<g, kRedThreads, 0, s>>>(static_cast<const float*>(amp), n, d_sets, nlow, nsets, d_terms, scratch, out);
  else
    k_pauli_sum<double><<<g, kRedThreads, 0, s>>>(static_cast<const double*>(amp), n, d_sets, nlow, nsets, d_terms, scratch, out);
  if (g > 1) return launch_sum_rows(scratch, 1, int(g), out, s);
  return cudaGetLastError();
}

}  // namespace nqpu
