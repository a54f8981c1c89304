// Runs of doublings on a block of warps: the window combination's chain of
// c (W - 1) dependent doublings, where nothing but the latency of one product
// after another counts.
//
// One Fp product per warp.  The two half-warps hold the 16 limbs of 28 bits
// (warp_field.cuh) one per lane and share the work: half h takes the partial
// products of eight limbs of a, then of its part of the fold, so a product
// issues 8 + 8 + 5 multiply-adds per lane against 65 in the layout of four
// products per warp; a lone warp issues one in 8 cycles on B200.  A level of a
// formula is four products of Fp, or of Fp2 as three of Fp each (Karatsuba),
// so a run takes 4 or 12 warps, which exchange results through shared memory.
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
// B200, per doubling: G1 2750 -> 2130 cycles, G2 5940 -> 3670 cycles
// against w_dbl.
#pragma once
#include "xyzz_warp.cuh"

namespace gm {

// Warps of a run and Fp products per field product
template <class F>
struct Chain;
template <>
struct Chain<Fp> {
  static constexpr int NS = 1, WARPS = 4;
};
template <>
struct Chain<Fp2> {
  static constexpr int NS = 3, WARPS = 12;
};

constexpr int CH_SCRATCH = 80;  // words per warp: a 16, b 32 (doubled), t 16, 16 unused by readers
constexpr int CH_SLOTS = 20;    // products whose results are kept
template <class F>
constexpr int chain_words() {
  return Chain<F>::WARPS * CH_SCRATCH + CH_SLOTS * Chain<F>::NS * 16;
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

// a b / R; a and b equal in both halves, the result in half 1.  Ranges as for
// w_redc; the result's limbs are not carried, in [-64, 2^29 + 64].
GM_DEVI int32_t c_mul(const ChainCtx &c, int32_t a, int32_t b) {
  int32_t *sa = c.scr, *sb = c.scr + 16, *st = c.scr + 48;
  sa[c.k] = a;  // the same word from both halves
  sb[c.k + 16 * c.h] = b;
  __syncwarp();
  const int4 a0 = reinterpret_cast<const int4 *>(sa)[2 * c.h], a1 = reinterpret_cast<const int4 *>(sa)[2 * c.h + 1];
  const int32_t av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
  const int32_t *pb = sb + 16 + c.k - 8 * c.h;
  const int nlo = c.k - 8 * c.h + 1;  // this lane's products that belong to the low column
  int64_t acc = 0, lo = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    acc += (int64_t)av[j] * pb[-j];
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

// n doublings of (X, Y) with L = 1, by the block's first Chain<F>::WARPS warps
// (all of them call it).  io: X, Y, L as WF<F>::LW limbs each in shared
// memory, read and written; work: chain_words<F>() words.
template <class F>
GM_DEVI void chain_dbl(int n, int32_t *io, int32_t *work) {
  constexpr int NS = Chain<F>::NS, NW = Chain<F>::WARPS, LW = WF<F>::LW;
  const int w = threadIdx.x >> 5;
  const int p = w / NS, s = w % NS;  // product of a level and its Fp factor
  const WarpTable &tab = w_table();
  ChainCtx c;
  c.k = threadIdx.x & 15;
  c.h = (threadIdx.x >> 4) & 1;
  c.scr = work + w * CH_SCRATCH;
#pragma unroll
  for (int j = 0; j < 8; j++) c.d[j] = 8 * c.h + j < W_FOLD ? tab.fold[min(8 * c.h + j, W_FOLD - 1)][c.k] : 0;
  c.p = tab.p[c.k];
  c.pa = c.k < 14 ? tab.p[c.k + 2] : 0;
  c.pb = c.k < 15 ? tab.p[c.k + 1] : 0;
  int32_t *raw = work + NW * CH_SCRATCH;
  auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); };
  // this warp's view of an Fp2 value: c0, c1 or c0 + c1
  auto view = [&](const int32_t *e) -> int32_t {
    if constexpr (NS == 1) return e[c.k];
    return s == 0 ? e[c.k] : s == 1 ? e[16 + c.k] : c_carry(c, e[c.k] + e[16 + c.k]);
  };
  auto put = [&](int slot, int32_t v) {
    if (c.h) raw[(slot * NS + s) * 16 + c.k] = v;
  };
  // view of the product in a slot, reduced for Fp2 (Karatsuba sums)
  auto get = [&](int slot) -> int32_t {
    const int32_t *r = raw + slot * NS * 16 + c.k;
    if constexpr (NS == 1) return r[0];
    const int32_t r0 = r[0], r1 = r[16], r2 = r[32];
    return c_reduce(c, s == 0 ? r0 - r1 : s == 1 ? r2 - r0 - r1 : r2 - 2 * r1);
  };
  auto mul4 = [&](int base, int np, int32_t a0, int32_t b0, int32_t a1, int32_t b1, int32_t a2, int32_t b2, int32_t a3,
                  int32_t b3) {
    if (p < np) {
      const int32_t a = p == 0 ? a0 : p == 1 ? a1 : p == 2 ? a2 : a3;
      const int32_t b = p == 0 ? b0 : p == 1 ? b1 : p == 2 ? b2 : b3;
      put(base + p, c_mul(c, a, b));
    }
    sync();
  };
  int32_t X = view(io), Y = view(io + LW), L = view(io + 2 * LW);
#pragma unroll 1
  while (n > 0) {
    int32_t U = 2 * Y;
    mul4(0, 4, X, X, U, U, U, Y, L, U);
    const int32_t V = get(1);
    int32_t h = get(2);
    L = get(3);
    const int32_t xx = get(0);
    int32_t M = c_reduce(c, 3 * xx);
    mul4(4, 3, M, M, X, V, V, h, 0, 0);
    const int32_t S = get(5), E = get(6);
    X = c_reduce(c, get(4) - 2 * S);
    mul4(8, 2, M, S - X, X, X, 0, 0, 0, 0);
    Y = c_reduce(c, get(8) - E);
    n--;
    if (n == 0) break;
    M = c_reduce(c, 3 * get(9));
    U = 2 * Y;
    mul4(12, 4, U, Y, M, M, M, 3 * X, L, U);
    h = get(12);
    const int32_t MM = get(13), MX = get(14);
    L = get(15);
    mul4(16, 4, X, h, MM, M, MX, h, h, h);
    X = c_reduce(c, MM - 4 * c_carry(c, get(16)));
    Y = c_reduce(c, 2 * c_carry(c, get(18)) - get(17) - 2 * c_carry(c, get(19)));
    n--;
  }
  // the views of c0 and c1 go back
  if (p == 0 && s < 2 && c.h == 0 && (NS > 1 || s == 0)) {
    io[s * 16 + c.k] = X;
    io[LW + s * 16 + c.k] = Y;
    io[2 * LW + s * 16 + c.k] = L;
  }
  sync();
}

}  // namespace gm
