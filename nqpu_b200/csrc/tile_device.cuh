// Device code shared by the tiled pass kernel and the batched executor: the
// shared-memory swizzle, register-block op bodies, op dispatch, the stage
// executor and async-copy helpers.  Included by .cu files only.
#pragma once
#include "sv_device.cuh"
#include "tileprog.h"

namespace nqpu {

constexpr int kTileThreads = 256;
constexpr int kVecPerThread = 16;
// Tile bits above the contiguous low block: k - c <= 8 (c >= 5 for complex64,
// c >= 4 for complex128, k <= 13 / 12), so the high-offset table has <= 256 entries.
constexpr int kHiOffBits = 8;
constexpr int kHiOffEntries = 1 << kHiOffBits;

__device__ __forceinline__ uint32_t swz(uint32_t u) {
  uint32_t w = u >> 3;
  uint32_t f = w ^ (w >> 3) ^ (w >> 6) ^ (w >> 9) ^ (w >> 12);
  return u ^ (f & 7u);
}

template <typename C>
__device__ __forceinline__ C csel(bool p, C a, C b) {
  C r;
  r.x = p ? a.x : b.x;
  r.y = p ? a.y : b.y;
  return r;
}

// ---- register-block op bodies (B, B0, B1, CB, ... are register-bit indices)
// Every amplitude index i below is a compile-time constant after unrolling, so
// the register block stays in registers; runtime register bits are turned into
// template arguments by the dispatch switches.

template <typename Real>
__device__ __forceinline__ void ldc2(const Real* __restrict__ p, typename Tr<Real>::C& a,
                                     typename Tr<Real>::C& b);
template <>
__device__ __forceinline__ void ldc2<float>(const float* __restrict__ p, float2& a, float2& b) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
template <>
__device__ __forceinline__ void ldc2<double>(const double* __restrict__ p, double2& a, double2& b) {
  a = *reinterpret_cast<const double2*>(p);
  b = *(reinterpret_cast<const double2*>(p) + 1);
}

// complex64 dense 2x2 on the pairs whose register bits CM (controls) are set
template <int NA, int B, int CM>
__device__ __forceinline__ void rb_u1(float2 (&a)[NA], float2 m0, float2 m1, float2 m2, float2 m3) {
  const PackedC p0 = pack_coef(m0), p1 = pack_coef(m1), p2 = pack_coef(m2), p3 = pack_coef(m3);
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if ((i & (1 << B)) || (i & CM) != CM) continue;
    const int j = i | (1 << B);
    const float2 x = a[i], y = a[j];
    const float2 sx = swap_ri(x), sy = swap_ri(y);
    float2 ti = __fmul2_rn(p0.p, x), tj = __fmul2_rn(p2.p, x);
    ti = __ffma2_rn(p0.q, sx, ti);
    tj = __ffma2_rn(p2.q, sx, tj);
    ti = __ffma2_rn(p1.p, y, ti);
    tj = __ffma2_rn(p3.p, y, tj);
    a[i] = __ffma2_rn(p1.q, sy, ti);
    a[j] = __ffma2_rn(p3.q, sy, tj);
  }
}

// The dense 2x2 on the pairs whose register bits CM (controls) are set.  FEW:
// complex128 at 128 registers has no room for the entries, and the spills land on
// every instruction of the stage loop: it reads them again for every pair
// (volatile, or the compiler would keep them).
template <typename Real, typename C, int NA, int B, int CM, bool FEW>
__device__ __forceinline__ void rb_u1_at(C (&a)[NA], const Real* mp) {
  if constexpr (FEW) {
    const volatile Real* m = mp;
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      if ((i & (1 << B)) || (i & CM) != CM) continue;
      C &x = a[i], &y = a[i | (1 << B)];
      C u, v;
      { const Real r = m[0], s = m[1]; u.x = r * x.x - s * x.y; u.y = r * x.y + s * x.x; }
      { const Real r = m[2], s = m[3]; u.x += r * y.x - s * y.y; u.y += r * y.y + s * y.x; }
      { const Real r = m[4], s = m[5]; v.x = r * x.x - s * x.y; v.y = r * x.y + s * x.x; }
      { const Real r = m[6], s = m[7]; v.x += r * y.x - s * y.y; v.y += r * y.y + s * y.x; }
      x = u;
      y = v;
    }
  } else {
    C m0, m1, m2, m3;
    ldc2<Real>(mp, m0, m1);
    ldc2<Real>(mp + 4, m2, m3);
    if constexpr (sizeof(Real) == 4) {
      rb_u1<NA, B, CM>(a, m0, m1, m2, m3);
    } else {
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        if ((i & (1 << B)) || (i & CM) != CM) continue;
        C &x = a[i], &y = a[i | (1 << B)];
        const C u = cmac2(m0, x, m1, y);
        y = cmac2(m2, x, m3, y);
        x = u;
      }
    }
  }
}

// The same with its control a run-time value: selects per amplitude.
template <typename Real, typename C, int NA, int B>
__device__ __forceinline__ void rb_u1_ctrl(C (&a)[NA], const Real* mp, bool tc, uint32_t creg) {
  C m0, m1, m2, m3;
  ldc2<Real>(mp, m0, m1);
  ldc2<Real>(mp + 4, m2, m3);
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (1 << B)) continue;
    const int j = i | (1 << B);
    const bool cond = tc && ((uint32_t(i) & creg) == creg);
    const C x = a[i], y = a[j];
    a[i] = csel(cond, cmac2(m0, x, m1, y), x);
    a[j] = csel(cond, cmac2(m2, x, m3, y), y);
  }
}

template <typename C, int NA>
__device__ __forceinline__ void rb_x1_generic(C (&a)[NA], int b, bool tc, uint32_t creg) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
#pragma unroll
    for (int bb = 0; bb < 5; ++bb) {
      if ((1 << bb) >= NA) break;
      if (bb != b) continue;
      if (i & (1 << bb)) continue;
      const int j = i | (1 << bb);
      const bool cond = tc && ((uint32_t(i) & creg) == creg);
      const C x = a[i], y = a[j];
      a[i] = csel(cond, y, x);
      a[j] = csel(cond, x, y);
    }
  }
}

// X on register bit B, controlled by the register bits CM (compile time) and
// by controls outside the registers (tc): per-thread selects (a register renaming
// where tc is always true is what only straight-line code can afford).
template <typename C, int NA, int B, int CM>
__device__ __forceinline__ void rb_x1_fixed(C (&a)[NA], bool tc) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (1 << B)) continue;
    if ((i & CM) != CM) continue;
    const int j = i | (1 << B);
    const C x = a[i], y = a[j];
    a[i] = csel(tc, y, x);
    a[j] = csel(tc, x, y);
  }
}

template <typename C, int NA, int NRB, int B>
__device__ __forceinline__ void dispatch_x1_ctrl(C (&a)[NA], uint32_t creg, bool tc) {
  switch (creg) {
#define NQ_X1C(V) case (V == 0 ? 0 : (1 << (V - 1))): \
    if constexpr (V == 0 || (V - 1 < NRB && V - 1 != B)) rb_x1_fixed<C, NA, B, (V == 0 ? 0 : (1 << (V - 1)))>(a, tc); break;
    NQ_X1C(0) NQ_X1C(1) NQ_X1C(2) NQ_X1C(3) NQ_X1C(4) NQ_X1C(5)
#undef NQ_X1C
    default: break;
  }
}

// real rotation as three shears in place (t = tan(phi / 2), s = sin(phi))
template <typename C, int NA, int B>
__device__ __forceinline__ void rb_rot(C (&a)[NA], decltype(C::x) t, decltype(C::x) s) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (1 << B)) continue;
    C &x = a[i], &y = a[i | (1 << B)];
    if constexpr (sizeof(t) == 4) {
      const float2 nt = make_float2(-t, -t), ss = make_float2(s, s);
      x = __ffma2_rn(nt, y, x);
      y = __ffma2_rn(ss, x, y);
      x = __ffma2_rn(nt, y, x);
    } else {
      x.x = fma(-t, y.x, x.x);
      x.y = fma(-t, y.y, x.y);
      y.x = fma(s, x.x, y.x);
      y.y = fma(s, x.y, y.y);
      x.x = fma(-t, y.x, x.x);
      x.y = fma(-t, y.y, x.y);
    }
  }
}

// RX(2 phi): the rotation of (x.re, y.im) by -phi and of (x.im, y.re) by phi
template <typename C, int NA, int B>
__device__ __forceinline__ void rb_cross(C (&a)[NA], decltype(C::x) t, decltype(C::x) s) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (1 << B)) continue;
    C &x = a[i], &y = a[i | (1 << B)];
    x.x = fma(t, y.y, x.x);
    x.y = fma(-t, y.x, x.y);
    y.y = fma(-s, x.x, y.y);
    y.x = fma(s, x.y, y.x);
    x.x = fma(t, y.y, x.x);
    x.y = fma(-t, y.x, x.y);
  }
}

// m * x in place, scalar: four operations and no re/im swap
template <typename C>
__device__ __forceinline__ void cmul_in(C m, C& v) {
  const auto u = m.y * v.y, w = m.y * v.x;
  v.x = fma(m.x, v.x, -u);
  v.y = fma(m.x, v.y, w);
}

// phase m on the register amplitudes whose bits CMASK are all set
template <typename C, int NA, int CMASK>
__device__ __forceinline__ void rb_ph(C (&a)[NA], C m) {
#pragma unroll
  for (int i = 0; i < NA; ++i)
    if ((i & CMASK) == CMASK) cmul_in(m, a[i]);
}

// one phase per register amplitude
template <typename Real, typename C, int NA>
__device__ __forceinline__ void rb_table(C (&a)[NA], const uint4* q) {
#pragma unroll
  for (int i = 0; i < NA; i += 2) {
    C u, v;
    ldc2<Real>(reinterpret_cast<const Real*>(q) + 2 * i, u, v);
    cmul_in(u, a[i]);
    cmul_in(v, a[i + 1]);
  }
}

// a phase as three shears in place: p.x = tan(alpha / 2), p.y = sin(alpha)
template <typename C>
__device__ __forceinline__ void turn_in(C p, C& v) {
  v.x = fma(-p.x, v.y, v.x);
  v.y = fma(p.y, v.x, v.y);
  v.x = fma(-p.x, v.y, v.x);
}
template <typename C, int NA, int CMASK>
__device__ __forceinline__ void rb_turn(C (&a)[NA], C p) {
#pragma unroll
  for (int i = 0; i < NA; ++i)
    if ((i & CMASK) == CMASK) turn_in(p, a[i]);
}
template <typename Real, typename C, int NA>
__device__ __forceinline__ void rb_turn_table(C (&a)[NA], const uint4* q) {
  if constexpr (sizeof(Real) == 4) {
#pragma unroll
    for (int i = 0; i < NA; i += 2) {
      C u, v;
      ldc2<Real>(reinterpret_cast<const Real*>(q) + 2 * i, u, v);
      turn_in(u, a[i]);
      turn_in(v, a[i + 1]);
    }
  } else {
    const volatile Real* m = reinterpret_cast<const volatile Real*>(q);  // not hoisted: no registers for it
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      C u;
      u.x = m[2 * i];
      u.y = m[2 * i + 1];
      turn_in(u, a[i]);
    }
  }
}

// sign flip (s = 0 or the sign bit) of the register amplitudes with bits CMASK
template <typename C, int NA, int CMASK>
__device__ __forceinline__ void rb_sign(C (&a)[NA], uint32_t s) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if ((i & CMASK) != CMASK) continue;
    if constexpr (sizeof(a[0].x) == 4) {
      a[i].x = __uint_as_float(__float_as_uint(a[i].x) ^ s);
      a[i].y = __uint_as_float(__float_as_uint(a[i].y) ^ s);
    } else {
      a[i].x = __hiloint2double(__double2hiint(a[i].x) ^ int(s), __double2loint(a[i].x));
      a[i].y = __hiloint2double(__double2hiint(a[i].y) ^ int(s), __double2loint(a[i].y));
    }
  }
}

// diag(d0, d1) on register bit B
template <typename C, int NA, int B>
__device__ __forceinline__ void rb_d1(C (&a)[NA], C d0, C d1) {
#pragma unroll
  for (int i = 0; i < NA; ++i) cmul_in((i & (1 << B)) ? d1 : d0, a[i]);
}
template <typename C, int NA, int B>
__device__ __forceinline__ void rb_turn1(C (&a)[NA], C p0, C p1) {
#pragma unroll
  for (int i = 0; i < NA; ++i) turn_in((i & (1 << B)) ? p1 : p0, a[i]);
}

// dense 4x4 on register bits (B0 = sub-index bit 0, B1 = bit 1); matrix rows
// are read from the op record (L1-resident) per quad to keep registers free.
template <typename Real, typename C, int NA, int B0, int B1, bool FEW>
__device__ __forceinline__ void rb_u2(C (&a)[NA], const Real* __restrict__ mp, bool tc, uint32_t creg) {
  constexpr int M0 = 1 << B0, M1 = 1 << B1;
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (M0 | M1)) continue;
    const bool cond = tc && ((uint32_t(i) & creg) == creg);
    const C x0 = a[i], x1 = a[i | M0], x2 = a[i | M1], x3 = a[i | M0 | M1];
    C y[4];
    if constexpr (!FEW) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        C m[4];
        ldc2<Real>(mp + 8 * r, m[0], m[1]);
        ldc2<Real>(mp + 8 * r + 4, m[2], m[3]);
        y[r] = cmac4(m, x0, x1, x2, x3);
      }
    } else {
      // one entry at a time: no room for a row
      auto mac = [&](int k, const C& x, C& acc) {
        const volatile Real* m = mp + 2 * k;  // read again per quad, not kept
        const Real r = m[0], s = m[1];
        acc.x = fma(r, x.x, fma(-s, x.y, acc.x));
        acc.y = fma(r, x.y, fma(s, x.x, acc.y));
      };
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        y[r].x = y[r].y = 0;
        mac(4 * r, x0, y[r]);
        mac(4 * r + 1, x1, y[r]);
        mac(4 * r + 2, x2, y[r]);
        mac(4 * r + 3, x3, y[r]);
      }
    }
    a[i] = csel(cond, y[0], x0);
    a[i | M0] = csel(cond, y[1], x1);
    a[i | M1] = csel(cond, y[2], x2);
    a[i | M0 | M1] = csel(cond, y[3], x3);
  }
}

template <typename C, int NA, int B0, int B1>
__device__ __forceinline__ void rb_sw(C (&a)[NA], bool tc, uint32_t creg) {
  constexpr int M0 = 1 << B0, M1 = 1 << B1;
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    if (i & (M0 | M1)) continue;
    const bool cond = tc && ((uint32_t(i) & creg) == creg);
    const C x1 = a[i | M0], x2 = a[i | M1];
    a[i | M0] = csel(cond, x2, x1);
    a[i | M1] = csel(cond, x1, x2);
  }
}

// ---- dispatch helpers ------------------------------------------------------
#define NQ_REG_CASES(M, ...) M(0, __VA_ARGS__) M(1, __VA_ARGS__) M(2, __VA_ARGS__) M(3, __VA_ARGS__) M(4, __VA_ARGS__)

template <typename Real, typename C, int NA, int NRB, int B0, bool FEW>
__device__ __forceinline__ void dispatch_u2_b(C (&a)[NA], int b1, const Real* mp, bool tc, uint32_t creg) {
  switch (b1) {
#define NQ_U2B(V) case V: if constexpr (V < NRB && V != B0) rb_u2<Real, C, NA, B0, V, FEW>(a, mp, tc, creg); break;
    NQ_U2B(0) NQ_U2B(1) NQ_U2B(2) NQ_U2B(3) NQ_U2B(4)
#undef NQ_U2B
    default: break;
  }
}

template <typename C, int NA, int NRB, int B0>
__device__ __forceinline__ void dispatch_sw_b(C (&a)[NA], int b1, bool tc, uint32_t creg) {
  switch (b1) {
#define NQ_SWB(V) case V: if constexpr (V < NRB && V != B0) rb_sw<C, NA, B0, V>(a, tc, creg); break;
    NQ_SWB(0) NQ_SWB(1) NQ_SWB(2) NQ_SWB(3) NQ_SWB(4)
#undef NQ_SWB
    default: break;
  }
}

// The other ops: 1q gates with register controls, X with register controls in
// the middle of a stage, SWAP and 4x4 matrices.  Their fields come in the header
// (warp-uniform, as the code): a record of its own behind it cost a second
// dependent read per op and 160 bytes of a program that shared memory may not hold
// (96 controlled unitaries on 8 qubits, complex64: 73 us, now 61).
template <typename Real, int NA, int NRB, bool FEW>
__device__ __forceinline__ void apply_op(typename Tr<Real>::C (&a)[NA], uint32_t kind, uint32_t fields, uint32_t cnr,
                                         const Real* mp, uint32_t vbase) {
  using C = typename Tr<Real>::C;
  const uint32_t rb0 = fields & 0xFFu, rb1 = (fields >> 8) & 0xFFu, creg = fields >> 16;
  const bool tc = (vbase & cnr) == cnr;
  switch (kind) {
    case OP_U1: {
      if constexpr (FEW) {  // four variants per bit would spill 44 bytes: one-qubit gates on 23 qubits 666 against 613 us
        switch (rb0) {
#define NQ_U1C(B, _) case B: if constexpr (B < NRB) rb_u1_ctrl<Real, C, NA, B>(a, mp, tc, creg); break;
          NQ_REG_CASES(NQ_U1C, 0)
#undef NQ_U1C
          default: break;
        }
        break;
      }
      // one register control (no gate has two on a dense target): only its half
      // of the pairs (8-qubit complex64 controlled unitaries 69 -> 61 us)
      if (!tc) break;
      switch (rb0 << 5 | creg) {
#define NQ_U1V(B, V) \
        case B << 5 | 1 << V: \
          if constexpr (B < NRB && V < NRB && B != V) rb_u1_at<Real, C, NA, B, 1 << V, FEW>(a, mp); \
          break;
#define NQ_U1C(B, _) NQ_U1V(B, 0) NQ_U1V(B, 1) NQ_U1V(B, 2) NQ_U1V(B, 3) NQ_U1V(B, 4)
        NQ_REG_CASES(NQ_U1C, 0)
#undef NQ_U1C
#undef NQ_U1V
        default: break;
      }
      break;
    }
    case OP_X1: {
      // X / CNOT kept in registers because later ops of the stage act on
      // its qubits (the others are deferred into the write-back map).  At
      // most one register control: a fixed register permutation; more
      // (Toffoli): generic per-amplitude selects.
      if (creg & (creg - 1)) {
        rb_x1_generic<C, NA>(a, int(rb0), tc, creg);
        break;
      }
      // selects even when tc is always true: a compile-time register
      // permutation here would make the allocator shuffle (and spill) the
      // register block on every other op's path
      switch (rb0) {
#define NQ_X1(B, _) case B: \
        if constexpr (B < NRB) dispatch_x1_ctrl<C, NA, NRB, B>(a, creg, tc); \
        break;
        NQ_REG_CASES(NQ_X1, 0)
#undef NQ_X1
        default: break;
      }
      break;
    }
    case OP_U2: {
      switch (rb0) {
#define NQ_U2A(B, _) case B: if constexpr (B < NRB) dispatch_u2_b<Real, C, NA, NRB, B, FEW>(a, rb1, mp, tc, creg); break;
        NQ_REG_CASES(NQ_U2A, 0)
#undef NQ_U2A
        default: break;
      }
      break;
    }
    case OP_SW: {
      switch (rb0) {
#define NQ_SWA(B, _) case B: if constexpr (B < NRB) dispatch_sw_b<C, NA, NRB, B>(a, rb1, tc, creg); break;
        NQ_REG_CASES(NQ_SWA, 0)
#undef NQ_SWA
        default: break;
      }
      break;
    }
    default:
      break;
  }
}

// The phase of a list of (mask, phase) entries for this thread; *p moves past it.
// complex64: exact sums of angles in 2^-32 turns and one sine / cosine, at any
// list length within about one rounding of the true phase (a running product of
// rounded factors would lose one per entry).  complex128: a product.
__device__ __forceinline__ uint32_t list_angle(const uint4*& p, uint32_t cnt, uint32_t angle, uint32_t vbase) {
  for (uint32_t i = 0; i < cnt; i += 2) {
    const uint4 e = *p++;
    if ((vbase & e.x) == e.x) angle += e.y;
    if ((vbase & e.z) == e.z) angle += e.w;  // an odd list ends in (0, 0)
  }
  return angle;
}
// The phase of an angle for cmul_in or, where every lane of the warp is within a
// quarter turn (*shear), for turn_in: a Trotter step's angles are, and there the
// shears keep the norm from drifting with the rounding of one (cos, sin) step after
// step.  Wider angles take the product: a shear would need a sign flip besides.
__device__ __forceinline__ float2 phase_of(uint32_t angle, bool* shear) {
  float s, c;
  sincospif(float(int32_t(angle)) * 0x1p-31f, &s, &c);
  *shear = __all_sync(0xffffffffu, c >= 0.0f);
  // c >= 0: the quotient is good to two roundings; an error in it turns the angle
  // by as much but leaves the shear's determinant
  return *shear ? make_float2(__fdividef(s, 1.0f + c), s) : make_float2(c, s);
}
__device__ __forceinline__ double2 list_phase(const uint4*& p, uint32_t cnt, double2 v, uint32_t vbase) {
  for (uint32_t i = 0; i < cnt; ++i, p += 2) {
    const uint32_t m = p->x;
    const double2 f = *reinterpret_cast<const double2*>(p + 1);
    if ((vbase & m) == m) v = cmul(f, v);
  }
  return v;
}

template <typename Real, int NA, int NRB>
__device__ __forceinline__ void rotate_bits(typename Tr<Real>::C (&a)[NA], uint32_t bits, const uint4& h,
                                            const uint4* q, bool cross) {
  using C = typename Tr<Real>::C;
  auto par = [&](int b) {  // t, s of bit b
    C v;
    if constexpr (sizeof(Real) == 4) {
      if (b == 0) v = make_float2(__uint_as_float(h.z), __uint_as_float(h.w));
      else v = reinterpret_cast<const float2*>(q)[b - 1];
    } else {
      v = reinterpret_cast<const double2*>(q)[b];
    }
    return v;
  };
#define NQ_ROT(B, _) \
  if constexpr (B < NRB) { \
    if (bits & (1u << B)) { \
      const C v = par(B); \
      if (cross) rb_cross<C, NA, B>(a, v.x, v.y); \
      else rb_rot<C, NA, B>(a, v.x, v.y); \
    } \
  }
  NQ_REG_CASES(NQ_ROT, 0)
#undef NQ_ROT
}

// Run a stage's program (tileprog.h) on the thread's register block.
// vbase = virtual index of register amplitude 0 (register bits are zero in it).
// Whole warps run it: the headers are made warp-uniform values, so that the
// dispatch compiles to uniform branches.
template <typename Real, int NA, int NRB, bool FEW>
__device__ __forceinline__ void apply_stage_prog(typename Tr<Real>::C (&a)[NA], const uint4* p,
                                                 const uint4* const end, uint32_t vbase) {
  using C = typename Tr<Real>::C;
  constexpr bool F32 = sizeof(Real) == 4;
  while (p < end) {
    uint4 h = *p;
    const uint4* q = p + 1;
    h.x = __shfl_sync(0xffffffffu, h.x, 0);
    const uint32_t code = h.x & 0xFFu, arg = (h.x >> 8) & 0xFFu;
    p += max(h.x >> 16, 1u);  // ends on any contents
    if (code <= TC_X) {
      const uint32_t bits = __shfl_sync(0xffffffffu, h.y, 0);
      if (code == TC_R) rotate_bits<Real, NA, NRB>(a, bits, h, q, false);
      else rotate_bits<Real, NA, NRB>(a, bits, h, q, true);
    } else if (code <= TC_T) {
      if (code == TC_TS) rb_turn_table<Real, C, NA>(a, q);
      else rb_table<Real, C, NA>(a, q);
    } else if (code <= TC_PU) {
      C d;
      bool shear = code == TC_PS;  // (no PS in complex128: its registers)
      if constexpr (F32) {
        if (code == TC_PH) d = phase_of(list_angle(q, h.y, h.z, vbase), &shear);
        else d = make_float2(__uint_as_float(h.z), __uint_as_float(h.w));
      } else {
        d = *reinterpret_cast<const double2*>(q);
        if (code == TC_PH) d = list_phase(++q, h.y, d, vbase);
      }
      switch (arg) {
#define NQ_A(V) \
        case V: \
          if constexpr (V < (1 << NRB)) { \
            if constexpr (F32) { \
              if (shear) rb_turn<C, NA, V>(a, d); \
              else rb_ph<C, NA, V>(a, d); \
            } else { \
              rb_ph<C, NA, V>(a, d); \
            } \
          } \
          break;
#define NQ_SETS(M) M(0) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(14) M(15) \
        M(16) M(17) M(18) M(19) M(20) M(21) M(22) M(23) M(24) M(25) M(26) M(27) M(28) M(29) M(30) M(31)
        NQ_SETS(NQ_A)
#undef NQ_A
        default: break;
      }
    } else if (code <= TC_SL) {
      uint32_t sign = 1u;
      if (code == TC_SL) {
        sign = h.z;
        for (uint32_t i = 0; i < h.y; i += 4) {
          const uint4 e = *q++;
          sign += (vbase & e.x) == e.x;
          if (i + 1 < h.y) sign += (vbase & e.y) == e.y;
          if (i + 2 < h.y) sign += (vbase & e.z) == e.z;
          if (i + 3 < h.y) sign += (vbase & e.w) == e.w;
        }
      }
      sign <<= 31;
      switch (arg) {
#define NQ_A(V) case V: if constexpr (V < (1 << NRB)) rb_sign<C, NA, V>(a, sign); break;
        NQ_SETS(NQ_A)
#undef NQ_A
#undef NQ_SETS
        default: break;
      }
    } else if (code == TC_D) {
      C d0, d1;
      bool shear = false;
      if constexpr (F32) {
        const uint32_t g = list_angle(q, h.y & 0xFFFFu, h.z, vbase), g1 = list_angle(q, h.y >> 16, g + h.w, vbase);
        float s, c;  // both as shears or both as products
        sincospif(float(int32_t(g)) * 0x1p-31f, &s, &c);
        d0 = make_float2(c, s);
        sincospif(float(int32_t(g1)) * 0x1p-31f, &s, &c);
        d1 = make_float2(c, s);
        shear = __all_sync(0xffffffffu, fminf(d0.x, d1.x) >= 0.0f);
        if (shear) {
          d0.x = __fdividef(d0.y, 1.0f + d0.x);
          d1.x = __fdividef(d1.y, 1.0f + d1.x);
        }
      } else {
        d0 = *reinterpret_cast<const double2*>(q);
        d1 = *reinterpret_cast<const double2*>(q + 1);
        q += 2;
        d0 = list_phase(q, h.y & 0xFFFFu, d0, vbase);
        d1 = cmul(d0, list_phase(q, h.y >> 16, d1, vbase));
      }
      switch (arg) {
#define NQ_B(B, _) \
        case B: \
          if constexpr (B < NRB) { \
            if (F32 && shear) rb_turn1<C, NA, B>(a, d0, d1); \
            else rb_d1<C, NA, B>(a, d0, d1); \
          } \
          break;
        NQ_REG_CASES(NQ_B, 0)
#undef NQ_B
        default: break;
      }
    } else if (code == TC_G) {
      const Real* m = reinterpret_cast<const Real*>(q);
      const bool tc = (vbase & h.y) == h.y;  // controls outside the registers
      switch (arg) {
#define NQ_B(B, _) \
        case B: \
          if constexpr (B < NRB) { \
            if (tc) rb_u1_at<Real, C, NA, B, 0, FEW>(a, m); \
          } \
          break;
        NQ_REG_CASES(NQ_B, 0)
#undef NQ_B
        default: break;
      }
    } else {
      apply_op<Real, NA, NRB, FEW>(a, arg, __shfl_sync(0xffffffffu, h.y, 0), h.z, reinterpret_cast<const Real*>(q), vbase);
    }
  }
}

template <typename Real>
__device__ __forceinline__ void unpack_vec(const typename Tr<Real>::V& v, typename Tr<Real>::C* a);
template <>
__device__ __forceinline__ void unpack_vec<float>(const float4& v, float2* a) {
  a[0] = make_float2(v.x, v.y);
  a[1] = make_float2(v.z, v.w);
}
template <>
__device__ __forceinline__ void unpack_vec<double>(const double2& v, double2* a) {
  a[0] = v;
}
template <typename Real>
__device__ __forceinline__ typename Tr<Real>::V pack_vec(const typename Tr<Real>::C* a);
template <>
__device__ __forceinline__ float4 pack_vec<float>(const float2* a) {
  return make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
}
template <>
__device__ __forceinline__ double2 pack_vec<double>(const double2* a) {
  return a[0];
}
template <typename Real>
__device__ __forceinline__ typename Tr<Real>::V pack_vec(typename Tr<Real>::C lo, typename Tr<Real>::C hi) {
  typename Tr<Real>::C t[2] = {lo, hi};
  return pack_vec<Real>(t);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Global amplitude index of tile-local index 0 of `tile` (tile id bit j -> qout[j]).
__device__ __forceinline__ uint64_t tile_base(const PassRec& P, uint64_t tile) {
  uint64_t base = 0;
  for (int j = 0; j < P.n_out; ++j)
    if ((tile >> j) & 1ull) base |= 1ull << P.qout[j];
  return base;
}


// Addressing of a full tile's copies between HBM and shared memory (KMAX tile
// bits, the usual contiguous low block): vector tid + i * threads sits at slot
// swz(tid) ^ swz(i * threads), and its HBM offset is the thread's part plus a
// combination of the four highest tile qubits, so a vector costs about five
// instructions beside the access (some twenty when every vector works out its
// own index and swizzle; two of three instructions of a one-stage pass).
template <typename Real, int KMAX>
struct TileCopy {
  static constexpr int VB = Tr<Real>::kVecBit;
  static constexpr int C = sizeof(Real) == 4 ? 5 : 4;
  static constexpr uint32_t kThreads = 1u << (KMAX - VB - 4);
  using V = typename Tr<Real>::V;

  static __host__ __device__ __forceinline__ bool fits(const PassRec& P) { return P.k == KMAX && P.c == C; }
  // f(slot, pointer) for each of the thread's 16 vectors; `base` = amplitude
  // index of the tile's first amplitude.
  template <typename F>
  static __device__ __forceinline__ void each(Real* amp, const PassRec& P, const uint64_t* hi_off, uint64_t base, F&& f) {
    uint32_t tid = threadIdx.x;
    asm volatile("" : "+r"(tid));  // worked out per tile: no registers held across the stages
    const uint32_t t = tid << VB;
    const uint32_t s0 = swz(tid);
    char* g = reinterpret_cast<char*>(amp) +
              (base + (t & ((1u << C) - 1u)) + hi_off[t >> C]) * (2 * sizeof(Real));
    const int top = KMAX - C - 4;
    const uint64_t d0 = uint64_t(2 * sizeof(Real)) << P.qhi[top], d1 = uint64_t(2 * sizeof(Real)) << P.qhi[top + 1];
    const uint64_t d2 = uint64_t(2 * sizeof(Real)) << P.qhi[top + 2], d3 = uint64_t(2 * sizeof(Real)) << P.qhi[top + 3];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      char* gh = g + ((h & 1) ? d2 : 0) + ((h & 2) ? d3 : 0);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const uint32_t i = uint32_t(4 * h + l);
        f(s0 ^ swz(i * kThreads), reinterpret_cast<V*>(gh + ((l & 1) ? d0 : 0) + ((l & 2) ? d1 : 0)));
      }
    }
  }
};

// Copy a pass's stage tables (StageTab, tileprog.h) and, behind them, the first
// `words` words of its program into shared memory, asynchronously: every thread
// of the CTA calls it, then waits for its copies (cp_async_wait0) and the CTA
// meets at a barrier.
__device__ __forceinline__ void load_pass_prog(const PassRec& P, const uint4* __restrict__ progs, int words,
                                               uint4* dst) {
  const uint4* src = progs + P.prog_begin;
  const int n = (P.stage_end - P.stage_begin) * (kStageTabWords / 4) + words;
  for (int i = threadIdx.x; i < n; i += blockDim.x) cp_async16(dst + i, src + i);
  cp_async_commit();
}

// Run stages [P.stage_begin, P.stage_end) of a pass on the tile held in shared
// memory `sv` (swizzled vector slots), with the pass's stage tables in `tabs`.
// Every thread of the CTA must call it (it contains block barriers); warps
// beyond nvec/16 threads only take part in them, and in a warp that is only partly
// needed the other lanes run along on an earlier thread's amplitudes without
// writing.  FEW: complex128 with too few registers to keep matrices in (rb_u1_at).
template <typename Real, bool FEW>
__device__ __forceinline__ void run_tile_stages(typename Tr<Real>::V* __restrict__ sv, const PassRec& P,
                                                const uint32_t* __restrict__ tabs,
                                                const uint4* prog, uint32_t ext) {
  using T = Tr<Real>;
  using C = typename T::C;
  constexpr int VB = T::kVecBit;
  constexpr int APV = T::kAmpsPerVec;
  constexpr int NA = kVecPerThread * APV;
  constexpr int NRB = VB + kRegFree;
  const int tid = threadIdx.x;
  const uint32_t active_threads = (1u << (P.k - VB)) / kVecPerThread;
  const int nst = P.stage_end - P.stage_begin;
  const uint32_t words = uint32_t(P.prog_words - nst * (kStageTabWords / 4));
  for (int si = 0; si < nst; ++si) {
    const uint32_t* Tb = tabs + si * kStageTabWords;
    if (uint32_t(tid & ~31) < active_threads) {
      const int tid_ = tid & int(active_threads - 1);
      const uint32_t ub = Tb[StageTab::UL + (tid_ & 15)] | Tb[StageTab::UH + (tid_ >> 4)];
      // swz is linear over XOR and ub, vm_i have disjoint bits, so
      // swz(ub | sum vm_i) = swz(ub) ^ xor_i swz(vm_i).
      const uint32_t sb = Tb[StageTab::SL + (tid_ & 15)] ^ Tb[StageTab::SH + (tid_ >> 4)];
      const uint4 sq = *reinterpret_cast<const uint4*>(Tb + StageTab::S);
      const uint32_t s0 = sq.x, s1 = sq.y, s2 = sq.z, s3 = sq.w;
      C a[NA];
#pragma unroll
      for (int r = 0; r < kVecPerThread; ++r) {
        const uint32_t slot = sb ^ ((r & 1) ? s0 : 0u) ^ ((r & 2) ? s1 : 0u) ^
                              ((r & 4) ? s2 : 0u) ^ ((r & 8) ? s3 : 0u);
        unpack_vec<Real>(sv[slot], a + r * APV);
      }
      const uint32_t vbase = (ub << VB) | ext;
      apply_stage_prog<Real, NA, NRB, FEW>(a, prog + Tb[StageTab::OB], prog + min(Tb[StageTab::OE], words), vbase);
      int wtid = threadIdx.x;  // read again: no register held across the program
      asm volatile("" : "+r"(wtid));
      if (uint32_t(wtid) < active_threads) {
        // Write-back through the stage's deferred permutation pi(p) = A p ^ w:
        // register amplitude p goes to the slot of logical index pi(p).  Slot
        // offsets are linear in the free register bits (register bits
        // VB..VB+3); for complex64, bit 0 of pi(p) selects the 8-byte half.
        uint32_t wslot = Tb[StageTab::WS], hw = Tb[StageTab::WH];
        const int nc = int(Tb[StageTab::NC]);
        for (int i = 0; i < nc; ++i) {
          const uint32_t cm = Tb[StageTab::CC + i];
          if ((vbase & cm) == cm) {
            wslot ^= Tb[StageTab::CS + i];
            hw ^= Tb[StageTab::CH + i];
          }
        }
        const uint4 cq = *reinterpret_cast<const uint4*>(Tb + StageTab::CW);
        const uint32_t c0 = cq.x, c1 = cq.y, c2 = cq.z, c3 = cq.w;
        const uint32_t sw = sb ^ wslot;
        if constexpr (VB == 1) {
          const uint32_t mz = Tb[StageTab::MZ], hb = Tb[StageTab::HB];
          const uint32_t h0 = hb & 1u, h1 = (hb >> 1) & 1u, h2 = (hb >> 2) & 1u, h3 = (hb >> 3) & 1u;
          if (mz == 1u) {
            // bit 0 stays bit 0: each vector keeps its pair, halves swap when
            // bit 0 of pi is flipped by the other register bits or by w
            if ((hb | hw) == 0u) {
              // no deferred flip of qubit 0 in this stage: whole vectors, no selects
#pragma unroll
              for (int r = 0; r < kVecPerThread; ++r) {
                const uint32_t slot = sw ^ ((r & 1) ? c0 : 0u) ^ ((r & 2) ? c1 : 0u) ^
                                      ((r & 4) ? c2 : 0u) ^ ((r & 8) ? c3 : 0u);
                sv[slot] = pack_vec<Real>(a[2 * r], a[2 * r + 1]);
              }
            } else {
#pragma unroll
              for (int r = 0; r < kVecPerThread; ++r) {
                const uint32_t slot = sw ^ ((r & 1) ? c0 : 0u) ^ ((r & 2) ? c1 : 0u) ^
                                      ((r & 4) ? c2 : 0u) ^ ((r & 8) ? c3 : 0u);
                const uint32_t hs = hw ^ ((r & 1) ? h0 : 0u) ^ ((r & 2) ? h1 : 0u) ^
                                    ((r & 4) ? h2 : 0u) ^ ((r & 8) ? h3 : 0u);
                const C lo = a[2 * r], hi = a[2 * r + 1];
                sv[slot] = hs ? pack_vec<Real>(hi, lo) : pack_vec<Real>(lo, hi);
              }
            }
          } else {
            // bit 0 moves into other bits: store each amplitude separately
            const uint32_t cz = Tb[StageTab::CZ], hz = Tb[StageTab::HZ];
            C* sa = reinterpret_cast<C*>(sv);
#pragma unroll
            for (int r = 0; r < kVecPerThread; ++r) {
              const uint32_t slot = sw ^ ((r & 1) ? c0 : 0u) ^ ((r & 2) ? c1 : 0u) ^
                                    ((r & 4) ? c2 : 0u) ^ ((r & 8) ? c3 : 0u);
              const uint32_t hs = hw ^ ((r & 1) ? h0 : 0u) ^ ((r & 2) ? h1 : 0u) ^
                                  ((r & 4) ? h2 : 0u) ^ ((r & 8) ? h3 : 0u);
              sa[2 * slot + hs] = a[2 * r];
              sa[2 * (slot ^ cz) + (hs ^ hz)] = a[2 * r + 1];
            }
          }
        } else {
#pragma unroll
          for (int r = 0; r < kVecPerThread; ++r) {
            const uint32_t slot = sw ^ ((r & 1) ? c0 : 0u) ^ ((r & 2) ? c1 : 0u) ^
                                  ((r & 4) ? c2 : 0u) ^ ((r & 8) ? c3 : 0u);
            sv[slot] = pack_vec<Real>(a + r * APV);
          }
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace nqpu
