// BLS12-446 base field Fp on sm_100a: 14 x 32-bit little-endian limbs.
//
// The limb layout is byte-identical to the reference's `Fp{uint64_t limb[7]}`
// (pdroalves/gpu_msm include/fp.h:13) on a little-endian machine, so device
// buffers cross the ABI without conversion.  Values are in Montgomery form with
// R = 2^448 (src/fp.cu:15-33).
//
// Montgomery multiplication is CIOS over 32-bit limbs on the IMAD pipe with PTX
// carry chains (mad.lo.cc / madc.hi.cc).  To keep one carry flag per chain,
// the partial products a_j*b_i are split by the parity of their column i + j
// into two accumulators, E (even columns) and O (odd columns).  A product's
// two words then always start at an even word of its accumulator, so the
// compiler makes one wide multiply-add of each mad.lo / madc.hi pair without
// moving registers about.  (Split by the parity of j, odd rows start pairs at
// odd words: 280 moves per product, and 2050 cycles a warp against 1810 at
// four warps per scheduler on B200; the multiplier's floor is 1640.)  Neither
// accumulator is shifted per iteration; the low column i is settled by
// tracking its exact carry c into column i+1, and the two halves are merged
// once at the end.  Per multiplication this is 2*14*14 product IMADs +
// 2*14*14 reduction IMADs + 14 quotient IMADs = 798.
//
// Two reduction modes:
//   * strict: inputs < p, output < p (canonical, bit-exact with the
//     reference's fp_mont_mul, src/fp.cu:370);
//   * lazy:   inputs < 2p, output < 2p (no final subtraction; valid because
//     4p < R).  Used inside point arithmetic; values are canonicalised before
//     any equality test and before leaving the device.
#pragma once
#include <cstdint>

#define GM_DEVI __device__ __forceinline__
#define GM_HDI __host__ __device__ __forceinline__

namespace gm {

constexpr int NL = 14;  // 32-bit limbs per Fp element

struct fp_t {
  uint32_t v[NL];
};

// Field constants as constexpr limb accessors: usable with compile-time
// indices (folded to immediates) and with run-time indices in device code.
struct FpConst {
  // p (src/fp.cu:15)
  GM_HDI static constexpr uint32_t P(int i) {
    switch (i) {
      case 0: return 0xaab0aaabu;
      case 1: return 0x311c0026u;
      case 2: return 0xc573b5ccu;
      case 3: return 0x56ee4528u;
      case 4: return 0xe23acdeeu;
      case 5: return 0x824e6dc3u;
      case 6: return 0xbac71602u;
      case 7: return 0x0f75a64bu;
      case 8: return 0x8a02fe32u;
      case 9: return 0x0095a4b7u;
      case 10: return 0x65aad640u;
      case 11: return 0x200fc349u;
      case 12: return 0x28c5e535u;
      case 13: return 0x3cdee0fbu;
      default: return 0u;
    }
  }
  // 2p
  GM_HDI static constexpr uint32_t P2(int i) {
    switch (i) {
      case 0: return 0x55615556u;
      case 1: return 0x6238004du;
      case 2: return 0x8ae76b98u;
      case 3: return 0xaddc8a51u;
      case 4: return 0xc4759bdcu;
      case 5: return 0x049cdb87u;
      case 6: return 0x758e2c05u;
      case 7: return 0x1eeb4c97u;
      case 8: return 0x1405fc64u;
      case 9: return 0x012b496fu;
      case 10: return 0xcb55ac80u;
      case 11: return 0x401f8692u;
      case 12: return 0x518bca6au;
      case 13: return 0x79bdc1f6u;
      default: return 0u;
    }
  }
  // R^2 mod p (src/fp.cu:21)
  GM_HDI static constexpr uint32_t R2(int i) {
    switch (i) {
      case 0: return 0xdc752b45u;
      case 1: return 0x2aff01ddu;
      case 2: return 0x421ccf5bu;
      case 3: return 0x92c772a7u;
      case 4: return 0xc347dad6u;
      case 5: return 0x140eef29u;
      case 6: return 0x22ea595eu;
      case 7: return 0xf5a1400cu;
      case 8: return 0xec145218u;
      case 9: return 0x99d91c9fu;
      case 10: return 0x90143d4bu;
      case 11: return 0x3bb6537fu;
      case 12: return 0x9be7974fu;
      case 13: return 0x3627854cu;
      default: return 0u;
    }
  }
  // R mod p = 1 in Montgomery form
  GM_HDI static constexpr uint32_t ONE(int i) {
    switch (i) {
      case 0: return 0x553d5554u;
      case 1: return 0x3b8fff65u;
      case 2: return 0xea3128cfu;
      case 3: return 0xa446eb5cu;
      case 4: return 0x7714c846u;
      case 5: return 0xf6c648f0u;
      case 6: return 0x14e3a7f5u;
      case 7: return 0xc22966d1u;
      case 8: return 0xd7f40737u;
      case 9: return 0xfda96d21u;
      case 10: return 0x6954a6ffu;
      case 11: return 0x7fc0f2dau;
      case 12: return 0x5ce86b2bu;
      case 13: return 0x0c847c13u;
      default: return 0u;
    }
  }
  // -p^-1 mod 2^32
  static constexpr uint32_t PINV = 0x0035fffdu;
};

// ---------------------------------------------------------------------------
// PTX carry-chain primitives.  `asm volatile` keeps the chain order; ptxas
// maps the PTX condition code onto carry predicates.
// ---------------------------------------------------------------------------
GM_DEVI uint32_t mad_lo_cc(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm volatile("mad.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
GM_DEVI uint32_t madc_lo_cc(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm volatile("madc.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
GM_DEVI uint32_t madc_hi_cc(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm volatile("madc.hi.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
GM_DEVI int64_t mad_wide(int32_t a, int32_t b, int64_t c) {
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
GM_DEVI uint32_t add_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GM_DEVI uint32_t addc_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GM_DEVI uint32_t addc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("addc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GM_DEVI uint32_t sub_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GM_DEVI uint32_t subc_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
GM_DEVI uint32_t subc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("subc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// ---------------------------------------------------------------------------
// Helpers on raw limb arrays
// ---------------------------------------------------------------------------

// r = a - m for the constant m = p (TWO_P = false) or 2p; returns borrow
template <bool TWO_P>
GM_DEVI uint32_t sub_const(uint32_t r[NL], const uint32_t a[NL]) {
  r[0] = sub_cc(a[0], TWO_P ? FpConst::P2(0) : FpConst::P(0));
#pragma unroll
  for (int i = 1; i < NL; i++) r[i] = subc_cc(a[i], TWO_P ? FpConst::P2(i) : FpConst::P(i));
  return subc(0, 0) & 1u;
}

// if a >= m: a -= m (constant-flow select), m = p or 2p
template <bool TWO_P>
GM_DEVI void cond_sub(uint32_t a[NL]) {
  uint32_t t[NL];
  const uint32_t borrow = sub_const<TWO_P>(t, a);
#pragma unroll
  for (int i = 0; i < NL; i++) a[i] = borrow ? a[i] : t[i];
}

// ---------------------------------------------------------------------------
// Montgomery multiplication (see header comment for the scheme).
// ---------------------------------------------------------------------------

// E, O += q * (get(0) .. get(13)) * 2^(32 i): even columns in E, odd columns in
// O, whose word k - 1 is column k.  The word above a chain was last written as
// the carry of an earlier row, so adding the carry to it cannot overflow.
template <class G>
GM_DEVI void mont_row(uint32_t (&E)[2 * NL + 2], uint32_t (&O)[2 * NL + 2], int i, uint32_t q, G get) {
  const int e = i & 1, o = 1 - e;  // first j of an even and of an odd column
  E[i + e] = mad_lo_cc(get(e), q, E[i + e]);
  E[i + e + 1] = madc_hi_cc(get(e), q, E[i + e + 1]);
#pragma unroll
  for (int j = e + 2; j < NL; j += 2) {
    E[i + j] = madc_lo_cc(get(j), q, E[i + j]);
    E[i + j + 1] = madc_hi_cc(get(j), q, E[i + j + 1]);
  }
  E[i + NL + e] = addc(E[i + NL + e], 0);
  O[i + o - 1] = mad_lo_cc(get(o), q, O[i + o - 1]);
  O[i + o] = madc_hi_cc(get(o), q, O[i + o]);
#pragma unroll
  for (int j = o + 2; j < NL; j += 2) {
    O[i + j - 1] = madc_lo_cc(get(j), q, O[i + j - 1]);
    O[i + j] = madc_hi_cc(get(j), q, O[i + j]);
  }
  O[i + NL - e] = addc(O[i + NL - e], 0);
}

// Quotient row i: makes column i 0 mod 2^32 and returns its exact carry into
// column i + 1 (c: the carry into column i).
GM_DEVI uint32_t mont_quotient_row(uint32_t (&E)[2 * NL + 2], uint32_t (&O)[2 * NL + 2], int i, uint32_t c) {
  const uint32_t u = (i == 0) ? E[0] : E[i] + O[i - 1] + c;
  mont_row(E, O, i, u * FpConst::PINV, [](int j) { return FpConst::P(j); });
  if (i == 0) return 0;  // E[0] == 0 exactly
  const uint32_t t = add_cc(E[i], O[i - 1]);
  const uint32_t c1 = addc(0, 0);
  (void)add_cc(t, c);
  return addc(c1, 0);
}

template <bool STRICT>
GM_DEVI void mont_mul_raw(uint32_t r[NL], const uint32_t a[NL], const uint32_t b[NL]) {
  uint32_t E[2 * NL + 2], O[2 * NL + 2];
#pragma unroll
  for (int k = 0; k < 2 * NL + 2; k++) {
    E[k] = 0;
    O[k] = 0;
  }
  uint32_t c = 0;  // exact carry out of the settled low columns
#pragma unroll
  for (int i = 0; i < NL; i++) {
    mont_row(E, O, i, b[i], [&](int j) { return a[j]; });
    c = mont_quotient_row(E, O, i, c);
  }
  // result = (E[14..27] + O[13..26] + c); higher words are 0 by the size bound
  r[0] = add_cc(E[NL], O[NL - 1]);
#pragma unroll
  for (int k = 1; k < NL; k++) r[k] = addc_cc(E[NL + k], O[NL - 1 + k]);
  r[0] = add_cc(r[0], c);
#pragma unroll
  for (int k = 1; k < NL; k++) r[k] = addc_cc(r[k], 0);
  if (STRICT) cond_sub<false>(r);
}

// ---------------------------------------------------------------------------
// Montgomery reduction of a 28-word value T < p * R: r = T * R^-1 mod p
// (below 2p before the optional final subtraction).  E holds the low half of
// T and the quotient products of even columns, O those of odd ones; the high
// half of T is added at the end.
// ---------------------------------------------------------------------------
template <bool STRICT>
GM_DEVI void redc_wide(uint32_t r[NL], const uint32_t T[2 * NL]) {
  uint32_t E[2 * NL + 2], O[2 * NL + 2];
#pragma unroll
  for (int k = 0; k < 2 * NL + 2; k++) {
    E[k] = k < NL ? T[k] : 0;
    O[k] = 0;
  }
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < NL; i++) c = mont_quotient_row(E, O, i, c);
  r[0] = add_cc(E[NL], O[NL - 1]);
#pragma unroll
  for (int k = 1; k < NL; k++) r[k] = addc_cc(E[NL + k], O[NL - 1 + k]);
  r[0] = add_cc(r[0], c);
#pragma unroll
  for (int k = 1; k < NL; k++) r[k] = addc_cc(r[k], 0);
  r[0] = add_cc(r[0], T[NL]);
#pragma unroll
  for (int k = 1; k < NL; k++) r[k] = addc_cc(r[k], T[NL + k]);
  if (STRICT) cond_sub<false>(r);
}

// ---------------------------------------------------------------------------
// Montgomery squaring (separated operand scanning): the 91 cross products
// a_i*a_j (i < j) are formed once, doubled by a one-bit shift, and the 14
// squares a_i^2 are added on the diagonal; the 28-word square is then reduced
// by the same 14 quotient rows as mont_mul_raw.  301 products instead of 392;
// measured 1.25x the throughput of mont_mul_raw(a, a) on B200 with identical
// (canonical) results.
//
// Cross products of row i go to two accumulators by the parity of j - i - 1
// (A: words 2i+1.., B: words 2i+2..), so each chain's words are disjoint and
// one carry flag suffices per chain.  A chain's carry-out word was last
// written as a previous chain's carry-out (value <= 1) or is still zero, so
// adding the carry never overflows.
// ---------------------------------------------------------------------------
template <bool STRICT>
GM_DEVI void mont_sqr_raw(uint32_t r[NL], const uint32_t a[NL]) {
  uint32_t A[2 * NL], B[2 * NL];
#pragma unroll
  for (int k = 0; k < 2 * NL; k++) {
    A[k] = 0;
    B[k] = 0;
  }
#pragma unroll
  for (int i = 0; i < NL - 1; i++) {
    {
      int j = i + 1;
      A[i + j] = mad_lo_cc(a[i], a[j], A[i + j]);
      A[i + j + 1] = madc_hi_cc(a[i], a[j], A[i + j + 1]);
      int top = i + j + 1;
#pragma unroll
      for (j = i + 3; j < NL; j += 2) {
        A[i + j] = madc_lo_cc(a[i], a[j], A[i + j]);
        A[i + j + 1] = madc_hi_cc(a[i], a[j], A[i + j + 1]);
        top = i + j + 1;
      }
      if (top + 1 < 2 * NL) A[top + 1] = addc(A[top + 1], 0);
    }
    if (i + 2 < NL) {
      int j = i + 2;
      B[i + j] = mad_lo_cc(a[i], a[j], B[i + j]);
      B[i + j + 1] = madc_hi_cc(a[i], a[j], B[i + j + 1]);
      int top = i + j + 1;
#pragma unroll
      for (j = i + 4; j < NL; j += 2) {
        B[i + j] = madc_lo_cc(a[i], a[j], B[i + j]);
        B[i + j + 1] = madc_hi_cc(a[i], a[j], B[i + j + 1]);
        top = i + j + 1;
      }
      if (top + 1 < 2 * NL) B[top + 1] = addc(B[top + 1], 0);
    }
  }
  // T = 2 (A + B) + diagonal; the cross sum is below 2^(2*448-1)
  uint32_t T[2 * NL];
  T[0] = add_cc(A[0], B[0]);
#pragma unroll
  for (int k = 1; k < 2 * NL; k++) T[k] = addc_cc(A[k], B[k]);
#pragma unroll
  for (int k = 2 * NL - 1; k > 0; k--) T[k] = __funnelshift_l(T[k - 1], T[k], 1);
  T[0] <<= 1;
  T[0] = mad_lo_cc(a[0], a[0], T[0]);
  T[1] = madc_hi_cc(a[0], a[0], T[1]);
#pragma unroll
  for (int i = 1; i < NL; i++) {
    T[2 * i] = madc_lo_cc(a[i], a[i], T[2 * i]);
    T[2 * i + 1] = madc_hi_cc(a[i], a[i], T[2 * i + 1]);
  }
  redc_wide<STRICT>(r, T);
}

// ---------------------------------------------------------------------------
// Field element API
// ---------------------------------------------------------------------------
struct Fp {
  using T = fp_t;
  static constexpr int LIMBS = NL;

  GM_DEVI static fp_t zero() {
    fp_t r;
#pragma unroll
    for (int i = 0; i < NL; i++) r.v[i] = 0;
    return r;
  }
  GM_DEVI static fp_t one() {
    fp_t r;
#pragma unroll
    for (int i = 0; i < NL; i++) r.v[i] = FpConst::ONE(i);
    return r;
  }
  GM_DEVI static bool is_zero_raw(const fp_t &a) {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < NL; i++) acc |= a.v[i];
    return acc == 0;
  }
  // a < 2p: a == 0 (mod p)
  GM_DEVI static bool is_zero(const fp_t &a) {
    uint32_t z = 0, q = 0;
#pragma unroll
    for (int i = 0; i < NL; i++) {
      z |= a.v[i];
      q |= a.v[i] ^ FpConst::P(i);
    }
    return z == 0 || q == 0;
  }
  // strict: a, b < p -> < p
  GM_DEVI static fp_t add(const fp_t &a, const fp_t &b) {
    fp_t r;
    r.v[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < NL; i++) r.v[i] = addc_cc(a.v[i], b.v[i]);
    cond_sub<false>(r.v);
    return r;
  }
  GM_DEVI static fp_t sub(const fp_t &a, const fp_t &b) {
    fp_t r;
    r.v[0] = sub_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < NL; i++) r.v[i] = subc_cc(a.v[i], b.v[i]);
    const uint32_t mask = 0u - (subc(0, 0) & 1u);
    r.v[0] = add_cc(r.v[0], FpConst::FpConst::P(0) & mask);
#pragma unroll
    for (int i = 1; i < NL; i++) r.v[i] = addc_cc(r.v[i], FpConst::P(i) & mask);
    return r;
  }
  GM_DEVI static fp_t dbl(const fp_t &a) { return add(a, a); }
  GM_DEVI static fp_t neg(const fp_t &a) {
    // p - a for a != 0, else 0 (src/fp.cu:436)
    if (is_zero_raw(a)) return a;
    fp_t r;
    r.v[0] = sub_cc(FpConst::FpConst::P(0), a.v[0]);
#pragma unroll
    for (int i = 1; i < NL; i++) r.v[i] = subc_cc(FpConst::P(i), a.v[i]);
    return r;
  }
  GM_DEVI static fp_t mul(const fp_t &a, const fp_t &b) {
    fp_t r;
    mont_mul_raw<true>(r.v, a.v, b.v);
    return r;
  }
  GM_DEVI static fp_t sqr(const fp_t &a) {
    fp_t r;
    mont_sqr_raw<true>(r.v, a.v);
    return r;
  }
  GM_DEVI static fp_t to_mont(const fp_t &a) {
    fp_t r2;
#pragma unroll
    for (int i = 0; i < NL; i++) r2.v[i] = FpConst::R2(i);
    return mul(a, r2);
  }
  GM_DEVI static fp_t from_mont(const fp_t &a) {
    fp_t o = zero();
    o.v[0] = 1;
    return mul(a, o);
  }
  GM_DEVI static fp_t small(uint32_t k) {  // k in Montgomery form
    fp_t t = zero();
    t.v[0] = k;
    return to_mont(t);
  }
  GM_DEVI static bool eq(const fp_t &a, const fp_t &b) {
    uint32_t d = 0;
#pragma unroll
    for (int i = 0; i < NL; i++) d |= a.v[i] ^ b.v[i];
    return d == 0;
  }
  // Montgomery-form inverse; 0 -> 0 (src/fp.cu:545)
  __device__ static fp_t inv(const fp_t &a);
};

// Same field with the multiplication out of line: one copy of the ~900
// instruction Montgomery product per kernel instead of one per call site.
// Operands and result travel in registers (no stack frame), and the loop body
// of the bucket accumulation then fits the instruction cache.
static __device__ __noinline__ fp_t fp_mul_call(fp_t a, fp_t b) {
  fp_t r;
  mont_mul_raw<true>(r.v, a.v, b.v);
  return r;
}
static __device__ __noinline__ fp_t fp_sqr_call(fp_t a) {
  fp_t r;
  mont_sqr_raw<true>(r.v, a.v);
  return r;
}

// a^-1 R^2 mod p, the inverse of a Montgomery-form element; 0 -> 0.  Division
// steps of Bernstein and Yang ("Fast constant-time gcd computation and modular
// inversion", 2019) on f = p, g = a: 28 steps depend on the low 28 bits of f
// and g alone and multiply (f, g) by a matrix over 2^28; the same matrix, with
// an exact division by 2^28 modulo p, acts on (d, e), kept at d a = f R^2 and
// e a = g R^2 modulo p.  16 limbs of 28 bits, plain 64-bit multiply-adds.
// delta starts at 1/2, which saves a round on average (33 against 34); 1288
// steps suffice for 446 bits from delta = 1 (their Theorem 11.2) and fewer
// from 1/2.  The work of 30 products (an exponentiation by p - 2 takes 600):
// 54 k cycles a warp on B200 with four warps per scheduler.  d and e grow by
// at most p / 2 a round, 25 p in all: the top limb stays below 2^31.
GM_HDI constexpr int32_t p28(int k) {  // limb k of p in 28-bit limbs
  const int j = (28 * k) / 32, s = (28 * k) % 32;
  const uint64_t w = (uint64_t)FpConst::P(j) | ((uint64_t)FpConst::P(j + 1) << 32);
  return (int32_t)((w >> s) & 0xfffffffull);
}
static __device__ __noinline__ fp_t fp_inv_call(fp_t a) {
  constexpr int N = 16;
  constexpr int32_t M28 = (1 << 28) - 1;
  int32_t f[N], g[N], d[N], e[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int j = (28 * k) / 32, s = (28 * k) % 32;
    f[k] = p28(k);
    d[k] = 0;
    g[k] = (int32_t)(__funnelshift_r(a.v[j], j + 1 < NL ? a.v[j + 1] : 0u, s) & (uint32_t)M28);
    e[k] = (int32_t)(__funnelshift_r(FpConst::R2(j), FpConst::R2(j + 1), s) & (uint32_t)M28);
  }
  int32_t delta = 0;  // the steps' delta - 1/2
#pragma unroll 1
  for (int it = 0; it < 47; it++) {
    int32_t any = 0;
#pragma unroll
    for (int k = 0; k < N; k++) any |= g[k];
    if (any == 0) break;
    uint32_t f0 = (uint32_t)f[0], g0 = (uint32_t)g[0];
    int32_t u = 1, v = 0, q = 0, r = 1;
    // 14 steps at a time, with a row of their matrix in one register: x 2^16 + y, |x| + |y| <= 2^14.
    // f and g are kept times 2^s: a step then adds 0, f or -f to g (a multiply-add), and doubles the new f.
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      uint32_t A = 1u << 16, B = 1u;
#pragma unroll
      for (int s = 0; s < 14; s++) {
        const bool odd = g0 & (1u << s), sw = odd && delta >= 0;
        const int32_t sg = sw ? -1 : (odd ? 1 : 0);
        const uint32_t f1 = sw ? g0 : f0, A1 = sw ? B : A;
        g0 += (uint32_t)(sg * (int32_t)f0);
        B += (uint32_t)(sg * (int32_t)A);
        f0 = f1 + f1;
        A = A1 + A1;
        delta = sw ? -delta : delta + 1;
      }
      f0 >>= 14;
      g0 >>= 14;
      const int32_t a1 = (int32_t)(A << 16) >> 16, a0 = (int32_t)(A - (uint32_t)a1) >> 16;
      const int32_t b1 = (int32_t)(B << 16) >> 16, b0 = (int32_t)(B - (uint32_t)b1) >> 16;
      const int32_t u1 = u, v1 = v;
      u = a0 * u1 + a1 * q;
      v = a0 * v1 + a1 * r;
      q = b0 * u1 + b1 * q;
      r = b0 * v1 + b1 * r;
    }
    // multiples of p that make the lowest limbs of d and e divisible, in [-2^27, 2^27)
    const int32_t md = (int32_t)((((uint32_t)u * (uint32_t)d[0] + (uint32_t)v * (uint32_t)e[0]) * FpConst::PINV) << 4) >> 4;
    const int32_t me = (int32_t)((((uint32_t)q * (uint32_t)d[0] + (uint32_t)r * (uint32_t)e[0]) * FpConst::PINV) << 4) >> 4;
    int64_t cf = 0, cg = 0, cd = 0, ce = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      const int32_t fk = f[k], gk = g[k], dk = d[k], ek = e[k];
      cf = mad_wide(v, gk, mad_wide(u, fk, cf));
      cg = mad_wide(r, gk, mad_wide(q, fk, cg));
      cd = mad_wide(md, p28(k), mad_wide(v, ek, mad_wide(u, dk, cd)));
      ce = mad_wide(me, p28(k), mad_wide(r, ek, mad_wide(q, dk, ce)));
      if (k > 0) {
        f[k - 1] = (int32_t)cf & M28;
        g[k - 1] = (int32_t)cg & M28;
        d[k - 1] = (int32_t)cd & M28;
        e[k - 1] = (int32_t)ce & M28;
      }
      cf >>= 28;
      cg >>= 28;
      cd >>= 28;
      ce >>= 28;
    }
    f[N - 1] = (int32_t)cf;
    g[N - 1] = (int32_t)cg;
    d[N - 1] = (int32_t)cd;
    e[N - 1] = (int32_t)ce;
  }
  // f is 1 or -1 (p for a = 0, where d = 0): +-d, brought into [0, p)
  const int32_t sg = f[0] == M28 ? -1 : 1;
  constexpr int64_t C = (int64_t)(((uint64_t)1 << 40) / ((uint64_t)p28(15) + 1));  // 2^40 / (p >> 420)
  const int32_t qd = (int32_t)(((int64_t)(sg * d[N - 1]) * C + ((int64_t)1 << 39)) >> 40);
  int64_t c = 0;
  uint64_t acc = 0;
  int bits = 0, j = 0;
  fp_t o;
#pragma unroll
  for (int k = 0; k < N; k++) {  // d - qd p + p lies in (0.4 p, 1.6 p)
    c += (int64_t)sg * d[k] + (int64_t)(1 - qd) * p28(k);
    acc |= (uint64_t)((uint32_t)c & (uint32_t)M28) << bits;
    c >>= 28;
    bits += 28;
    if (bits >= 32) {
      o.v[j++] = (uint32_t)acc;
      acc >>= 32;
      bits -= 32;
    }
  }
  cond_sub<false>(o.v);
  return o;
}
__device__ inline fp_t Fp::inv(const fp_t &a) { return fp_inv_call(a); }

struct FpOut : Fp {
  GM_DEVI static fp_t mul(const fp_t &a, const fp_t &b) { return fp_mul_call(a, b); }
  GM_DEVI static fp_t sqr(const fp_t &a) { return fp_sqr_call(a); }
};
// 16-byte vector loads/stores of field elements (56 B = 3.5 x 16 B, so
// records are laid out with 16-byte alignment by the packers).
GM_DEVI void load_fp_u64(fp_t &r, const uint64_t *src) {
#pragma unroll
  for (int i = 0; i < NL / 2; i++) {
    const uint64_t w = src[i];
    r.v[2 * i] = (uint32_t)w;
    r.v[2 * i + 1] = (uint32_t)(w >> 32);
  }
}
GM_DEVI void store_fp_u64(uint64_t *dst, const fp_t &a) {
#pragma unroll
  for (int i = 0; i < NL / 2; i++) dst[i] = (uint64_t)a.v[2 * i] | ((uint64_t)a.v[2 * i + 1] << 32);
}

}  // namespace gm
