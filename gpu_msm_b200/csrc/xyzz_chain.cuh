// Runs of doublings on a block of warps: the window combination's chain of
// c (W - 1) dependent doublings, where nothing but the latency of one product
// after another counts.
//
// One coefficient of one product per warp.  The two half-warps hold the 16
// limbs of 28 bits (warp_field.cuh) one per lane and share the work: half h
// takes the partial products of eight limbs of a, then of its part of the fold,
// so a product issues 8 + 8 + 5 multiply-adds per lane against 65 in the layout
// of four products per warp; a lone warp issues one in 8 cycles on B200.  A
// level of a formula is four products: 4 warps for Fp; 8 for Fp2, whose
// coefficients a0 b0 - a1 b1 and a0 b1 + a1 b0 are summed in columns and reduced
// once (Karatsuba on 12 warps put three on a scheduler and a recombination
// behind every level: 3670 cycles a doubling).  The warps exchange results
// through shared memory.
//
// Two doublings take 5 levels.  With U = 2Y, M = 3X^2, S = 4XY^2:
//   1  X^2, V = U^2, h = 2Y^2, L U      (L collects the Z factors 2Y)
//   2  M^2, S = X V, E = V h = 8Y^4     X' = M^2 - 2S
//   3  M (S - X'), X'^2                 Y' = M (S - X') - E,  M' = 3X'^2
//   4  h' = 2Y'^2, M'^2, 3M'X', L U'
//   5  d = X'h', M'^3, a = 3M'X'h', h'^2   X" = M'^2 - 4d,  Y" = 2a - M'^3 - 2h'^2
// (S' - X" = 3S' - M'^2 turns the last product of the second doubling into
// products that do not wait for X").  A run ends with ZZ L^2 and ZZZ L^3; a
// point of order two on the way shows as L = 0.
//
// B200, per doubling: G1 2750 -> 2030 cycles, G2 5940 -> 2840 cycles
// against w_dbl.
#pragma once
#include "xyzz_warp.cuh"

namespace gm {

struct CPair;

// Coefficients of a field element and warps of a run
template <class F>
struct Chain;
template <>
struct Chain<Fp> {
  using V = int32_t;
  static constexpr int NC = 1, WARPS = 4;
};
template <>
struct Chain<Fp2> {
  using V = CPair;
  static constexpr int NC = 2, WARPS = 8;
};

constexpr int CH_SLOTS = 20;  // products whose results are kept
// words per warp: a 16 and b 32 (doubled) per coefficient, t 16, 16 unused by readers
template <class F>
constexpr int ch_scratch() {
  return Chain<F>::NC * 48 + 32;
}
template <class F>
constexpr int chain_words() {
  return Chain<F>::WARPS * ch_scratch<F>() + CH_SLOTS * Chain<F>::NC * 16;
}

// This warp's place and constants in a run
struct ChainCtx {
  int k, h;         // limb and half of this lane
  int32_t d[8];     // fold constants of this lane's column, limbs 8h .. 8h + 7
  int32_t p, pa, pb;
  int32_t *scr;
};

GM_DEVI int32_t c_carry(const ChainCtx &c, int32_t v) {
  const int32_t up = __shfl_up_sync(0xffffffffu, v >> 28, 1, 16);
  return (c.k == 15 ? v : (v & WM28)) + (c.k == 0 ? 0 : up);
}
GM_DEVI int32_t c_reduce(const ChainCtx &c, int32_t v) {
  constexpr int64_t C = (int64_t)(((uint64_t)1 << 40) / ((uint64_t)p28(15) + 1));  // as in w_reduce
  const int32_t top = __shfl_sync(0xffffffffu, v, 15, 16);
  const int32_t q = (int32_t)(((int64_t)top * C + ((int64_t)1 << 39)) >> 40);
  return c_carry(c, v - q * c.p);
}

// One limb of each coefficient of an element: an integer, or a pair
struct CPair {
  int32_t x, y;
};
GM_DEVI CPair operator-(const CPair &a, const CPair &b) { return CPair{a.x - b.x, a.y - b.y}; }
GM_DEVI CPair operator*(int32_t k, const CPair &a) { return CPair{k * a.x, k * a.y}; }
GM_DEVI CPair c_carry(const ChainCtx &c, const CPair &v) { return CPair{c_carry(c, v.x), c_carry(c, v.y)}; }
GM_DEVI CPair c_reduce(const ChainCtx &c, const CPair &v) { return CPair{c_reduce(c, v.x), c_reduce(c, v.y)}; }
GM_DEVI void c_put(const ChainCtx &c, int32_t *e, int32_t v) { e[c.k] = v; }
GM_DEVI void c_put(const ChainCtx &c, int32_t *e, const CPair &v) {
  e[c.k] = v.x;
  e[16 + c.k] = v.y;
}
GM_DEVI void c_get(const ChainCtx &c, const int32_t *e, int32_t &v) { v = e[c.k]; }
GM_DEVI void c_get(const ChainCtx &c, const int32_t *e, CPair &v) { v = CPair{e[c.k], e[16 + c.k]}; }
GM_DEVI int32_t c_pick(int p, int32_t a0, int32_t a1, int32_t a2, int32_t a3) {
  return p == 0 ? a0 : p == 1 ? a1 : p == 2 ? a2 : a3;
}
GM_DEVI CPair c_pick(int p, const CPair &a0, const CPair &a1, const CPair &a2, const CPair &a3) {
  return CPair{c_pick(p, a0.x, a1.x, a2.x, a3.x), c_pick(p, a0.y, a1.y, a2.y, a3.y)};
}

// The factors of coefficient s to the warp's slots: a b, or a0 b0 + (-a1) b1
// (s = 0) and a0 b1 + a1 b0 (s = 1)
GM_DEVI void c_factors(const ChainCtx &c, int, int32_t *sa, int32_t *sb, int32_t a, int32_t b) {
  sa[c.k] = a;  // the same word from both halves
  sb[c.k + 16 * c.h] = b;
}
GM_DEVI void c_factors(const ChainCtx &c, int s, int32_t *sa, int32_t *sb, const CPair &a, const CPair &b) {
  sa[c.k] = a.x;
  sa[16 + c.k] = s ? a.y : -a.y;
  sb[c.k + 16 * c.h] = s ? b.y : b.x;
  sb[32 + c.k + 16 * c.h] = s ? b.x : b.y;
}

// Coefficient s of a b / R (a b / R itself for Fp); a and b equal in both
// halves, the result in half 1.  The columns stay below 2^63: for Fp limbs up
// to 2^29 + 64 in both factors, for Fp2 up to 2^28 + 8 in one and three times
// that in the other.  The result's limbs are not carried, in [-64, 2^29 + 64].
template <int NC, class V>
GM_DEVI int32_t c_mul(const ChainCtx &c, int s, const V &a, const V &b) {
  int32_t *sa = c.scr, *sb = c.scr + 16 * NC, *st = c.scr + 48 * NC;
  c_factors(c, s, sa, sb, a, b);
  __syncwarp();
  const int nlo = c.k - 8 * c.h + 1;  // this lane's products that belong to the low column
  int64_t acc = 0, lo = 0;
  int32_t av[NC][8];
#pragma unroll
  for (int n = 0; n < NC; n++) {
    const int4 a0 = reinterpret_cast<const int4 *>(sa + 16 * n)[2 * c.h];
    const int4 a1 = reinterpret_cast<const int4 *>(sa + 16 * n)[2 * c.h + 1];
    av[n][0] = a0.x, av[n][1] = a0.y, av[n][2] = a0.z, av[n][3] = a0.w;
    av[n][4] = a1.x, av[n][5] = a1.y, av[n][6] = a1.z, av[n][7] = a1.w;
  }
  const int32_t *pb = sb + 16 + c.k - 8 * c.h;
#pragma unroll
  for (int j = 0; j < 8; j++) {
#pragma unroll
    for (int n = 0; n < NC; n++) acc += (int64_t)av[n][j] * pb[32 * n - j];
    if (j < nlo) lo = acc;
  }
  const int64_t hi = acc - lo;
  // half 0 gets the low column, half 1 the high one
  const int64_t mine = (c.h ? hi : lo) + __shfl_xor_sync(0xffffffffu, c.h ? lo : hi, 16);
  int32_t x = (int32_t)mine & WM28, y = (int32_t)(mine >> 28) & WM28, z = (int32_t)(mine >> 56);
  int32_t y1 = __shfl_up_sync(0xffffffffu, y, 1, 16), z2 = __shfl_up_sync(0xffffffffu, z, 2, 16);
  if (c.k < 1) y1 = 0;
  if (c.k < 2) z2 = 0;
  st[c.k + 16 * c.h] = x + y1 + z2;  // half 0's are the limbs (14 and 15 meet d = 0)
  __syncwarp();
  // half 0: columns 14, 15 of the product; half 1: columns 16 .. 29
  int64_t f = c.h ? (c.k < 14 ? mine : 0) : (c.k < 14 ? 0 : mine + z2 + (c.k == 14 ? y1 : 0));
  const int4 t0 = reinterpret_cast<const int4 *>(st)[2 * c.h], t1 = reinterpret_cast<const int4 *>(st)[2 * c.h + 1];
  const int32_t tv[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
  for (int j = 0; j < 8; j++) f += (int64_t)tv[j] * c.d[j];  // d is 0 beyond limb 13
  f += __shfl_xor_sync(0xffffffffu, f, 16);
  int64_t v0 = __shfl_sync(0xffffffffu, f, 14, 16), v1 = __shfl_sync(0xffffffffu, f, 15, 16);
  constexpr uint64_t NP = w_np56();
  const uint64_t m = ((uint64_t)v0 + ((uint64_t)v1 << 28)) * NP;
  const int32_t m0 = (int32_t)(m & (uint64_t)WM28), m1 = (int32_t)((m >> 28) & (uint64_t)WM28);
  f = c.k < 14 ? f : (c.k == 14 ? mine : 0);
  f += (int64_t)m0 * c.pa;
  f += (int64_t)m1 * c.pb;
  v0 += (int64_t)m0 * p28(0);
  v1 += (int64_t)m0 * p28(1) + (int64_t)m1 * p28(0) + (v0 >> 28);
  if (c.k == 0) f += v1 >> 28;
  x = (int32_t)f & WM28;
  y = (int32_t)(f >> 28) & WM28;
  z = (int32_t)(f >> 56);
  y1 = __shfl_up_sync(0xffffffffu, c.k == 14 ? (int32_t)(f >> 28) : y, 1, 16);
  z2 = __shfl_up_sync(0xffffffffu, z, 2, 16);
  if (c.k < 1) y1 = 0;
  if (c.k < 2) z2 = 0;
  return x + y1 + z2;
}

// n doublings of (X, Y) with L = 1, by Chain<F>::WARPS warps of the block from
// warp w0 on (all of them call it; they share barrier 1).  io: X, Y, L as
// WF<F>::LW limbs each in shared memory, read and written; work:
// chain_words<F>() words.
//
// Ranges, in p: X, Y, M within 0.51; Fp products within (-0.5, 2), Fp2
// coefficients within (-1, 2).  Every c_reduce sees |v| < 7 and limbs that stay
// below 2^31 with the multiple of p added: sums of carried values up to 4 of
// one, and the products that are doubled at the end are carried or reduced first.
template <class F>
GM_DEVI void chain_dbl(int n, int w0, int32_t *io, int32_t *work) {
  constexpr int NC = Chain<F>::NC, NW = Chain<F>::WARPS, LW = WF<F>::LW;
  using V = typename Chain<F>::V;
  // (threadIdx.x >> 5 here: 2420 cycles a doubling against 2030 for G1, 3090 against 2840 for G2)
  const int w = w_warp() - w0;
  const int p = w / NC, s = w % NC;  // product of a level and its coefficient
  const WarpTable &tab = w_table();
  ChainCtx c;
  c.k = threadIdx.x & 15;
  c.h = (threadIdx.x >> 4) & 1;
  c.scr = work + w * ch_scratch<F>();
#pragma unroll
  for (int j = 0; j < 8; j++) c.d[j] = 8 * c.h + j < W_FOLD ? tab.fold[min(8 * c.h + j, W_FOLD - 1)][c.k] : 0;
  c.p = tab.p[c.k];
  c.pa = c.k < 14 ? tab.p[c.k + 2] : 0;
  c.pb = c.k < 15 ? tab.p[c.k + 1] : 0;
  int32_t *raw = work + NW * ch_scratch<F>();
  auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); };
  auto raw_get = [&](int slot) {
    V v;
    c_get(c, raw + slot * NC * 16, v);
    return v;
  };
  // a product as a factor of the next level (Fp2 factors are carried)
  auto factor = [&](const V &v) {
    if constexpr (NC == 1) return v;
    return c_carry(c, v);
  };
  auto get = [&](int slot) { return factor(raw_get(slot)); };
  // small enough to be taken four times
  auto small = [&](const V &v) {
    if constexpr (NC == 1) return c_carry(c, v);
    return c_reduce(c, v);
  };
  auto mul4 = [&](int base, int np, const V &a0, const V &b0, const V &a1, const V &b1, const V &a2, const V &b2,
                  const V &a3, const V &b3) {
    if (NC == 1 || p < np) {  // (Fp's four warps have a scheduler each: an idle one computes a product nobody reads)
      const int32_t r = c_mul<NC>(c, s, c_pick(p, a0, a1, a2, a3), c_pick(p, b0, b1, b2, b3));
      if (c.h) raw[((base + p) * NC + s) * 16 + c.k] = r;
    }
    sync();
  };
  V X, Y, L;
  c_get(c, io, X);
  c_get(c, io + LW, Y);
  c_get(c, io + 2 * LW, L);
  const V none{};
#pragma unroll 1
  while (n > 0) {
    V U = factor(2 * Y);
    mul4(0, 4, X, X, U, U, U, Y, L, U);
    const V Vv = get(1);
    V h = get(2);
    L = get(3);
    V M = c_reduce(c, 3 * raw_get(0));
    mul4(4, 3, M, M, X, Vv, Vv, h, none, none);
    const V S = get(5), E = raw_get(6);
    X = c_reduce(c, raw_get(4) - 2 * S);
    mul4(8, 2, M, S - X, X, X, none, none, none, none);
    Y = c_reduce(c, raw_get(8) - E);
    n--;
    if (n == 0) break;
    M = c_reduce(c, 3 * raw_get(9));
    U = factor(2 * Y);
    mul4(12, 4, U, Y, M, M, M, 3 * X, L, U);
    h = get(12);
    const V MM = get(13), MX = get(14);
    L = get(15);
    mul4(16, 4, X, h, MM, M, MX, h, h, h);
    X = c_reduce(c, MM - 4 * small(raw_get(16)));
    Y = c_reduce(c, 2 * small(raw_get(18)) - raw_get(17) - 2 * small(raw_get(19)));
    n--;
  }
  if (w == 0 && c.h == 0) {
    c_put(c, io, X);
    c_put(c, io + LW, Y);
    c_put(c, io + 2 * LW, L);
  }
  sync();
}

}  // namespace gm
