// Host-side BLS12-446 arithmetic for the C-ABI helpers that the reference runs
// on the CPU (pdroalves/gpu_msm rust-api/src/c_wrapper.cu:12-59, 261-288):
// Montgomery conversion, affine <-> projective, point-at-infinity helpers.
// 7 x 64-bit limbs, CIOS Montgomery multiplication with 128-bit products.
// All results are canonical (< p), so they agree with the reference's host
// functions bit for bit on canonical inputs.
#pragma once
#include <cstdint>
#include <cstring>

#include "../../include/gpu_msm_b200.h"

namespace gm_host {

typedef unsigned __int128 u128;
constexpr int L = 7;

static const uint64_t P[L] = {0x311c0026aab0aaabULL, 0x56ee4528c573b5ccULL, 0x824e6dc3e23acdeeULL,
                              0x0f75a64bbac71602ULL, 0x0095a4b78a02fe32ULL, 0x200fc34965aad640ULL,
                              0x3cdee0fb28c5e535ULL};
static const uint64_t R2[L] = {0x2AFF01DDDC752B45ULL, 0x92C772A7421CCF5BULL, 0x140EEF29C347DAD6ULL,
                               0xF5A1400C22EA595EULL, 0x99D91C9FEC145218ULL, 0x3BB6537F90143D4BULL,
                               0x3627854C9BE7974FULL};
static const uint64_t PINV64 = 0xcd63fd900035fffdULL;  // -p^-1 mod 2^64

inline bool geq_p(const uint64_t a[L]) {
  for (int i = L - 1; i >= 0; i--) {
    if (a[i] > P[i]) return true;
    if (a[i] < P[i]) return false;
  }
  return true;
}
inline void sub_p(uint64_t a[L]) {
  uint64_t br = 0;
  for (int i = 0; i < L; i++) {
    u128 d = (u128)a[i] - P[i] - br;
    a[i] = (uint64_t)d;
    br = (uint64_t)(d >> 64) ? 1 : 0;
  }
}
inline bool is_zero(const uint64_t a[L]) {
  uint64_t acc = 0;
  for (int i = 0; i < L; i++) acc |= a[i];
  return acc == 0;
}

// c = a*b*R^-1 mod p (CIOS, 64-bit words); canonical for canonical inputs
inline void mont_mul(uint64_t c[L], const uint64_t a[L], const uint64_t b[L]) {
  uint64_t t[L + 2] = {0};
  for (int i = 0; i < L; i++) {
    u128 carry = 0;
    for (int j = 0; j < L; j++) {
      carry += (u128)a[j] * b[i] + t[j];
      t[j] = (uint64_t)carry;
      carry >>= 64;
    }
    carry += t[L];
    t[L] = (uint64_t)carry;
    t[L + 1] = (uint64_t)(carry >> 64);
    const uint64_t m = t[0] * PINV64;
    carry = (u128)m * P[0] + t[0];
    carry >>= 64;
    for (int j = 1; j < L; j++) {
      carry += (u128)m * P[j] + t[j];
      t[j - 1] = (uint64_t)carry;
      carry >>= 64;
    }
    carry += t[L];
    t[L - 1] = (uint64_t)carry;
    t[L] = t[L + 1] + (uint64_t)(carry >> 64);
  }
  uint64_t r[L];
  for (int i = 0; i < L; i++) r[i] = t[i];
  if (t[L] || geq_p(r)) sub_p(r);
  memcpy(c, r, sizeof(r));
}

// c = a^2 R^-1 mod p: the 21 cross products once, doubled, plus the 7
// squares on the diagonal (28 products instead of 49), then the same
// word-by-word Montgomery reduction; canonical for canonical inputs.
inline void mont_sqr(uint64_t c[L], const uint64_t a[L]) {
  uint64_t t[2 * L + 1];
  memset(t, 0, sizeof(t));
  for (int i = 0; i < L - 1; i++) {
    u128 carry = 0;
    for (int j = i + 1; j < L; j++) {
      carry += (u128)a[i] * a[j] + t[i + j];
      t[i + j] = (uint64_t)carry;
      carry >>= 64;
    }
    t[i + L] = (uint64_t)carry;
  }
  uint64_t top = 0;
  for (int k = 0; k < 2 * L; k++) {
    const uint64_t nt = t[k] >> 63;
    t[k] = (t[k] << 1) | top;
    top = nt;
  }
  u128 carry = 0;
  for (int i = 0; i < L; i++) {
    const u128 sq = (u128)a[i] * a[i];
    carry += (u128)t[2 * i] + (uint64_t)sq;
    t[2 * i] = (uint64_t)carry;
    carry >>= 64;
    carry += (u128)t[2 * i + 1] + (uint64_t)(sq >> 64);
    t[2 * i + 1] = (uint64_t)carry;
    carry >>= 64;
  }
  for (int i = 0; i < L; i++) {
    const uint64_t m = t[i] * PINV64;
    u128 cy = 0;
    for (int j = 0; j < L; j++) {
      cy += (u128)m * P[j] + t[i + j];
      t[i + j] = (uint64_t)cy;
      cy >>= 64;
    }
    for (int k = i + L; cy != 0 && k < 2 * L + 1; k++) {
      cy += t[k];
      t[k] = (uint64_t)cy;
      cy >>= 64;
    }
  }
  uint64_t r[L];
  for (int i = 0; i < L; i++) r[i] = t[L + i];
  if (t[2 * L] || geq_p(r)) sub_p(r);
  memcpy(c, r, sizeof(r));
}

inline void add(uint64_t c[L], const uint64_t a[L], const uint64_t b[L]) {
  u128 carry = 0;
  uint64_t r[L];
  for (int i = 0; i < L; i++) {
    carry += (u128)a[i] + b[i];
    r[i] = (uint64_t)carry;
    carry >>= 64;
  }
  if (carry || geq_p(r)) sub_p(r);
  memcpy(c, r, sizeof(r));
}
inline void sub(uint64_t c[L], const uint64_t a[L], const uint64_t b[L]) {
  uint64_t r[L], br = 0;
  for (int i = 0; i < L; i++) {
    u128 d = (u128)a[i] - b[i] - br;
    r[i] = (uint64_t)d;
    br = (uint64_t)(d >> 64) ? 1 : 0;
  }
  if (br) {
    u128 carry = 0;
    for (int i = 0; i < L; i++) {
      carry += (u128)r[i] + P[i];
      r[i] = (uint64_t)carry;
      carry >>= 64;
    }
  }
  memcpy(c, r, sizeof(r));
}
inline void neg(uint64_t c[L], const uint64_t a[L]) {
  if (is_zero(a)) {
    memset(c, 0, sizeof(uint64_t) * L);
    return;
  }
  uint64_t t[L];
  memcpy(t, a, sizeof(t));
  sub(c, P, t);
}
inline void to_mont(uint64_t c[L], const uint64_t a[L]) { mont_mul(c, a, R2); }
inline void from_mont(uint64_t c[L], const uint64_t a[L]) {
  uint64_t one[L] = {1, 0, 0, 0, 0, 0, 0};
  mont_mul(c, a, one);
}
inline void one_mont(uint64_t c[L]) {
  uint64_t one[L] = {1, 0, 0, 0, 0, 0, 0};
  to_mont(c, one);
}
// a^-1 R^2 mod p, the inverse of a Montgomery-form element; 0 -> 0.  Division
// steps of Bernstein and Yang ("Fast constant-time gcd computation and modular
// inversion", 2019), delta from 1/2, as on the device (fp_inv_call of
// field.cuh): 62 steps depend on the low 62 bits of f and g and multiply (f, g)
// by a matrix over 2^62; the same matrix, with an exact division modulo p, acts
// on (d, e), kept at d a = f R^2 and e a = g R^2.  8 limbs of 62 bits, the top
// one signed; about 15 rounds.  One conversion of a projective G1 point took
// 46 us with an exponentiation by p - 2 and takes 4 us.
inline void mont_inv(uint64_t c[L], const uint64_t a_in[L]) {
  typedef __int128 i128;
  constexpr int N = 8;
  constexpr uint64_t M62 = (uint64_t(1) << 62) - 1;
  uint64_t a[L];
  memcpy(a, a_in, sizeof(a));
  while (geq_p(a)) sub_p(a);
  if (is_zero(a)) {
    memset(c, 0, sizeof(uint64_t) * L);
    return;
  }
  auto cut = [](int64_t *o, const uint64_t *v) {
    for (int k = 0; k < N; k++) {
      const int j = 62 * k / 64, s = 62 * k % 64;
      const u128 w = j < L ? (u128)v[j] | (u128)(j + 1 < L ? v[j + 1] : 0) << 64 : 0;
      o[k] = (int64_t)((uint64_t)(w >> s) & M62);
    }
  };
  int64_t p[N], f[N], g[N], d[N] = {0}, e[N];
  cut(p, P);
  cut(f, P);
  cut(g, a);
  cut(e, R2);
  int64_t delta = 0;  // the steps' delta - 1/2
  for (int it = 0; it < 22; it++) {  // 1288 steps suffice; 21 rounds hold more
    int64_t any = 0;
    for (int k = 0; k < N; k++) any |= g[k];
    if (any == 0) break;
    uint64_t f0 = (uint64_t)f[0], g0 = (uint64_t)g[0], u = 1, v = 0, q = 0, r = 1;
    for (int s = 0; s < 62; s++) {
      const uint64_t odd = 0 - (g0 & 1), sw = odd & ~(uint64_t)(delta >> 63);
      // swap: (f, g) -> (g, -f), then g + f where g was odd
      const uint64_t xf = (f0 ^ g0) & sw, xu = (u ^ q) & sw, xv = (v ^ r) & sw;
      f0 ^= xf;
      g0 = ((g0 ^ xf) ^ sw) - sw;
      u ^= xu;
      q = ((q ^ xu) ^ sw) - sw;
      v ^= xv;
      r = ((r ^ xv) ^ sw) - sw;
      delta = ((delta ^ (int64_t)sw) - (int64_t)sw) + (int64_t)(1 + sw);  // -delta, or delta + 1
      g0 = (g0 + (f0 & odd)) >> 1;
      q += u & odd;
      r += v & odd;
      u <<= 1;
      v <<= 1;
    }
    const int64_t su = (int64_t)u, sv = (int64_t)v, sq = (int64_t)q, sr = (int64_t)r;
    // multiples of p that make the lowest limbs of d and e divisible, in [-2^61, 2^61)
    const int64_t md = (int64_t)(((u * (uint64_t)d[0] + v * (uint64_t)e[0]) * PINV64) << 2) >> 2;
    const int64_t me = (int64_t)(((q * (uint64_t)d[0] + r * (uint64_t)e[0]) * PINV64) << 2) >> 2;
    i128 cf = 0, cg = 0, cd = 0, ce = 0;
    for (int k = 0; k < N; k++) {
      const int64_t fk = f[k], gk = g[k], dk = d[k], ek = e[k];
      cf += (i128)su * fk + (i128)sv * gk;
      cg += (i128)sq * fk + (i128)sr * gk;
      cd += (i128)su * dk + (i128)sv * ek + (i128)md * p[k];
      ce += (i128)sq * dk + (i128)sr * ek + (i128)me * p[k];
      if (k > 0) {
        f[k - 1] = (int64_t)((uint64_t)cf & M62);
        g[k - 1] = (int64_t)((uint64_t)cg & M62);
        d[k - 1] = (int64_t)((uint64_t)cd & M62);
        e[k - 1] = (int64_t)((uint64_t)ce & M62);
      }
      cf >>= 62;
      cg >>= 62;
      cd >>= 62;
      ce >>= 62;
    }
    f[N - 1] = (int64_t)cf;
    g[N - 1] = (int64_t)cg;
    d[N - 1] = (int64_t)cd;
    e[N - 1] = (int64_t)ce;
  }
  // f is 1 or -1: +-d, a value within +-12 p, brought into [0, p)
  const int64_t sg = f[0] == (int64_t)M62 ? -1 : 1;
  int64_t t[N];
  i128 cy = 0;
  for (int k = 0; k < N; k++) {  // + 16 p > 0
    cy += (i128)sg * d[k] + (i128)16 * p[k];
    t[k] = k < N - 1 ? (int64_t)((uint64_t)cy & M62) : (int64_t)cy;
    cy >>= 62;
  }
  for (int m = 16; m > 0; m >>= 1) {  // t < 32 p: subtract 16 p, 8 p, .. p where it fits
    int64_t w[N];
    cy = 0;
    for (int k = 0; k < N; k++) {
      cy += (i128)t[k] - (i128)m * p[k];
      w[k] = k < N - 1 ? (int64_t)((uint64_t)cy & M62) : (int64_t)cy;
      cy >>= 62;
    }
    if (w[N - 1] >= 0) memcpy(t, w, sizeof(t));
  }
  for (int k = 0; k < L; k++) {
    const int j = 64 * k / 62, s = 64 * k % 62;
    u128 w = (u128)(uint64_t)t[j] | (u128)(j + 1 < N ? (uint64_t)t[j + 1] : 0) << 62;
    if (s) {
      w >>= s;
      if (j + 2 < N) w |= (u128)(uint64_t)t[j + 2] << (124 - s);
    }
    c[k] = (uint64_t)w;
  }
}

// Fp2 (i^2 = -1)
inline void fp2_mul(Fp2 &c, const Fp2 &a, const Fp2 &b) {
  uint64_t t0[L], t1[L], s0[L], s1[L], t2[L];
  mont_mul(t0, a.c0.limb, b.c0.limb);
  mont_mul(t1, a.c1.limb, b.c1.limb);
  add(s0, a.c0.limb, a.c1.limb);
  add(s1, b.c0.limb, b.c1.limb);
  mont_mul(t2, s0, s1);
  sub(c.c0.limb, t0, t1);
  sub(c.c1.limb, t2, t0);
  sub(c.c1.limb, c.c1.limb, t1);
}
inline bool fp2_is_zero(const Fp2 &a) { return is_zero(a.c0.limb) && is_zero(a.c1.limb); }
inline void fp2_inv(Fp2 &c, const Fp2 &a) {
  if (fp2_is_zero(a)) {
    memset(&c, 0, sizeof(c));
    return;
  }
  uint64_t t0[L], t1[L], nrm[L], ni[L], na1[L];
  mont_mul(t0, a.c0.limb, a.c0.limb);
  mont_mul(t1, a.c1.limb, a.c1.limb);
  add(nrm, t0, t1);
  mont_inv(ni, nrm);
  Fp2 r;
  mont_mul(r.c0.limb, a.c0.limb, ni);
  neg(na1, a.c1.limb);
  mont_mul(r.c1.limb, na1, ni);
  c = r;
}

}  // namespace gm_host

// ---------------------------------------------------------------------------
// Host XYZZ arithmetic for the window combination of the blocking host-buffer
// calls (~300 doublings on the calling thread).  Same EFD formulas as xyzz.cuh:
// dbl-2008-s-1 and add-2008-s for a = 0, all values canonical (< p).
// ---------------------------------------------------------------------------
namespace gm_host {

struct HFp {
  uint64_t v[L];
};
struct HFp2 {
  HFp c0, c1;
};

struct F1 {
  using T = HFp;
  static constexpr int WORDS = L;
  static void zero(T &a) { memset(a.v, 0, sizeof(a.v)); }
  static bool is_zero(const T &a) { return gm_host::is_zero(a.v); }
  static void add(T &c, const T &a, const T &b) { gm_host::add(c.v, a.v, b.v); }
  static void sub(T &c, const T &a, const T &b) { gm_host::sub(c.v, a.v, b.v); }
  static void mul(T &c, const T &a, const T &b) { gm_host::mont_mul(c.v, a.v, b.v); }
  static void sqr(T &c, const T &a) { gm_host::mont_sqr(c.v, a.v); }
};

struct F2 {
  using T = HFp2;
  static constexpr int WORDS = 2 * L;
  static void zero(T &a) { memset(&a, 0, sizeof(a)); }
  static bool is_zero(const T &a) { return gm_host::is_zero(a.c0.v) && gm_host::is_zero(a.c1.v); }
  static void add(T &c, const T &a, const T &b) {
    gm_host::add(c.c0.v, a.c0.v, b.c0.v);
    gm_host::add(c.c1.v, a.c1.v, b.c1.v);
  }
  static void sub(T &c, const T &a, const T &b) {
    gm_host::sub(c.c0.v, a.c0.v, b.c0.v);
    gm_host::sub(c.c1.v, a.c1.v, b.c1.v);
  }
  static void mul(T &c, const T &a, const T &b) {
    uint64_t t0[L], t1[L], s0[L], s1[L], t2[L];
    mont_mul(t0, a.c0.v, b.c0.v);
    mont_mul(t1, a.c1.v, b.c1.v);
    gm_host::add(s0, a.c0.v, a.c1.v);
    gm_host::add(s1, b.c0.v, b.c1.v);
    mont_mul(t2, s0, s1);
    gm_host::sub(c.c0.v, t0, t1);
    gm_host::sub(c.c1.v, t2, t0);
    gm_host::sub(c.c1.v, c.c1.v, t1);
  }
  // (a0 + a1 i)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 i
  static void sqr(T &c, const T &a) {
    uint64_t s[L], d[L], m[L];
    gm_host::add(s, a.c0.v, a.c1.v);
    gm_host::sub(d, a.c0.v, a.c1.v);
    mont_mul(m, a.c0.v, a.c1.v);
    mont_mul(c.c0.v, s, d);
    gm_host::add(c.c1.v, m, m);
  }
};

template <class F>
struct HXyzz {
  typename F::T X, Y, ZZ, ZZZ;
};

template <class F>
inline bool hx_is_inf(const HXyzz<F> &p) {
  return F::is_zero(p.ZZ);
}

template <class F>
inline void hx_dbl(HXyzz<F> &p) {
  using T = typename F::T;
  if (hx_is_inf(p)) return;
  T U, V, W, S, xx, M, t, X3, Y3;
  F::add(U, p.Y, p.Y);
  F::mul(V, U, U);
  F::mul(W, U, V);
  F::mul(S, p.X, V);
  F::mul(xx, p.X, p.X);
  F::add(M, xx, xx);
  F::add(M, M, xx);
  F::mul(X3, M, M);
  F::add(t, S, S);
  F::sub(X3, X3, t);
  F::sub(t, S, X3);
  F::mul(Y3, M, t);
  F::mul(t, W, p.Y);
  F::sub(Y3, Y3, t);
  F::mul(p.ZZ, V, p.ZZ);
  F::mul(p.ZZZ, W, p.ZZZ);
  p.X = X3;
  p.Y = Y3;
}

template <class F>
inline void hx_add(HXyzz<F> &acc, const HXyzz<F> &q) {
  using T = typename F::T;
  if (hx_is_inf(q)) return;
  if (hx_is_inf(acc)) {
    acc = q;
    return;
  }
  T U1, U2, S1, S2, P, R, PP, PPP, Q, X3, Y3, t;
  F::mul(U1, acc.X, q.ZZ);
  F::mul(U2, q.X, acc.ZZ);
  F::mul(S1, acc.Y, q.ZZZ);
  F::mul(S2, q.Y, acc.ZZZ);
  F::sub(P, U2, U1);
  F::sub(R, S2, S1);
  if (F::is_zero(P)) {
    if (F::is_zero(R)) {
      hx_dbl(acc);
    } else {
      F::zero(acc.X);
      F::zero(acc.Y);
      F::zero(acc.ZZ);
      F::zero(acc.ZZZ);
    }
    return;
  }
  F::mul(PP, P, P);
  F::mul(PPP, P, PP);
  F::mul(Q, U1, PP);
  F::mul(X3, R, R);
  F::sub(X3, X3, PPP);
  F::add(t, Q, Q);
  F::sub(X3, X3, t);
  F::sub(t, Q, X3);
  F::mul(Y3, R, t);
  F::mul(t, S1, PPP);
  F::sub(Y3, Y3, t);
  F::mul(t, acc.ZZ, q.ZZ);
  F::mul(acc.ZZ, t, PP);
  F::mul(t, acc.ZZZ, q.ZZZ);
  F::mul(acc.ZZZ, t, PPP);
  acc.X = X3;
  acc.Y = Y3;
}

// Jacobian coordinates (x = X/Z^2, y = Y/Z^3) for the runs of c doublings
// of the Horner loop: dbl-2009-l for a = 0 costs 2M + 5S against 6M + 3S
// in XYZZ.  XYZZ -> Jacobian without an inversion: Z' = ZZZ,
// X' = X ZZ^2, Y' = Y ZZZ^2 (since ZZZ^2 = ZZ^3); back: ZZ = Z^2, ZZZ = Z^3.
template <class F>
struct HJac {
  typename F::T X, Y, Z;
};

template <class F>
inline void jac_from_xyzz(HJac<F> &j, const HXyzz<F> &p) {
  typename F::T t;
  F::sqr(t, p.ZZ);
  F::mul(j.X, p.X, t);
  F::sqr(t, p.ZZZ);
  F::mul(j.Y, p.Y, t);
  j.Z = p.ZZZ;
}

template <class F>
inline void xyzz_from_jac(HXyzz<F> &p, const HJac<F> &j) {
  p.X = j.X;
  p.Y = j.Y;
  F::sqr(p.ZZ, j.Z);
  F::mul(p.ZZZ, p.ZZ, j.Z);
}

// 2P in place (dbl-2009-l); Y = 0 or Z = 0 gives Z = 0 (infinity)
template <class F>
inline void jac_dbl(HJac<F> &j) {
  using T = typename F::T;
  T A, B, C, D, E, Fv, t;
  F::sqr(A, j.X);
  F::sqr(B, j.Y);
  F::sqr(C, B);
  F::add(t, j.X, B);
  F::sqr(D, t);
  F::sub(D, D, A);
  F::sub(D, D, C);
  F::add(D, D, D);
  F::add(E, A, A);
  F::add(E, E, A);
  F::sqr(Fv, E);
  F::mul(t, j.Y, j.Z);
  F::add(j.Z, t, t);
  F::add(t, D, D);
  F::sub(j.X, Fv, t);
  F::sub(t, D, j.X);
  F::mul(j.Y, E, t);
  F::add(C, C, C);
  F::add(C, C, C);
  F::add(C, C, C);
  F::sub(j.Y, j.Y, C);
}

// Horner with XYZZ doublings only (dbl-2008-s-1): the reference point for
// gm_host_selftest's check of the Jacobian version below.
template <class F>
inline void horner_xyzz(HXyzz<F> &res, const HXyzz<F> *sums, int W, int c) {
  memset(&res, 0, sizeof(res));
  for (int w = W - 1; w >= 0; w--) {
    if (!hx_is_inf(res))
      for (int k = 0; k < c; k++) hx_dbl(res);
    hx_add(res, sums[w]);
  }
}

// result = sum_w 2^(c w) S_w (Horner, MSB first), then to homogeneous
// projective (X*ZZZ, Y*ZZ, ZZ*ZZZ); infinity -> all zero.  `sums` holds W
// device-layout XYZZ points (32-bit limb order == 64-bit limb order on a
// little-endian host); `out` receives 3 coordinates of F::WORDS u64.
template <class F>
inline void horner_to_proj(uint64_t *out, const HXyzz<F> *sums, int W, int c) {
  HXyzz<F> res;
  memset(&res, 0, sizeof(res));
  HJac<F> j;
  for (int w = W - 1; w >= 0; w--) {
    if (!hx_is_inf(res)) {
      jac_from_xyzz(j, res);
      for (int k = 0; k < c; k++) jac_dbl(j);
      xyzz_from_jac(res, j);
    }
    hx_add(res, sums[w]);
  }
  typename F::T X, Y, Z;
  if (hx_is_inf(res)) {
    memset(out, 0, 3 * F::WORDS * sizeof(uint64_t));
    return;
  }
  F::mul(X, res.X, res.ZZZ);
  F::mul(Y, res.Y, res.ZZ);
  F::mul(Z, res.ZZ, res.ZZZ);
  memcpy(out, &X, F::WORDS * 8);
  memcpy(out + F::WORDS, &Y, F::WORDS * 8);
  memcpy(out + 2 * F::WORDS, &Z, F::WORDS * 8);
}

}  // namespace gm_host
