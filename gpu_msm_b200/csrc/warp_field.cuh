// Field arithmetic spread over a warp, for the phases where a few dependent
// point operations decide the time (small MSMs, the upper levels of the
// bucket reduction, the fix-up of straddling buckets, the window
// combination).
//
// Layout.  A warp is four groups of eight lanes; a group holds one Fp element
// as 16 limbs of 28 bits, lane l the limbs 2l and 2l + 1, signed 32-bit and
// redundant (a few units outside [0, 2^28)); the top limb is kept whole, so
// it carries the sign.  16 x 28 = 448, so R = 2^448 and the Montgomery form
// are those of memory.  All four groups hold the same operands, each computes
// one of up to four products of a formula level, and shuffles hand the results round.
//
// Why.  One thread's Montgomery product issues 400 32x32->64 multiply-adds,
// 4 cycles each on the multiplier of a warp scheduler, in one carry chain:
// 1600 cycles at the least and about 2900 measured on B200.  28-bit limbs
// need no carry flags (16 products of 2^29 x 2^29 stay below 2^62), so a lane
// adds up its two columns with plain 64-bit multiply-adds, 32 for the
// product and 33 for the reduction, and the four products of a level take
// the time of one.  The serial chain of a full XYZZ addition, 4 products,
// fell from about 20 us in four lanes of one product each to under 2 us.  At
// full occupancy an addition costs 260 multiplier slots of a warp against 175
// for one addition per thread, so the phases that fill the GPU with
// independent additions stay on one thread per addition.
//
// Product.  Columns T_k = sum a_i b_(k-i) of the pair (2l, 2l+1), low half
// and high half (columns +16), from shared-memory copies of a (read by all
// lanes at once) and b (doubled, so that a rotated read needs no wrap).
// Reduction by 2^-392 with one matrix product: the 14 low limbs t_k (after
// one carry pass) times D_k = 2^(28 k - 392) mod p, added to T_14..T_31; then
// two Montgomery digits, m = -V p^-1 mod 2^56, and a shift by 2^56, which is
// one lane: lane 7 holds columns 0 and 1 of V, lane l < 7 columns 2l + 2 and
// 2l + 3, so the shifted result is in place.  For |a| < A p, |b| < B p the
// result lies in (-0.24 A B p, (0.24 A B + 1) p), congruent to a b / R.
//
// Contract: all 32 lanes of a warp call these functions together, with
// operands that are equal in the four groups except where a function says
// "per group".  Kernels call w_setup once, at block start, and are launched
// with w_smem_bytes<F>(warps) bytes of dynamic shared memory.
#pragma once
#include "fp2.cuh"

namespace gm {

constexpr int32_t WM28 = (1 << 28) - 1;
constexpr int W_FOLD = 14;  // limbs folded by the matrix product

struct WarpTable {
  int32_t fold[W_FOLD][16];  // D_k limbs in lane order: pair l = limbs 2l+2, 2l+3; pair 7 = limbs 0, 1
  int32_t p[16];             // p
  int32_t pm[8][4];          // per lane: p[2l+1], p[2l+2], p[2l+3], 0; lane 7: p[15], p[0], p[1], 0
};

constexpr WarpTable make_warp_table() {
  WarpTable t{};
  uint32_t v[NL] = {1};
  for (int k = W_FOLD - 1; k >= 0; k--) {
    for (int s = 0; s < 28; s++) {  // v = v / 2 mod p
      uint64_t cy = 0;
      const uint32_t odd = v[0] & 1u;
      for (int i = 0; i < NL; i++) {
        cy += (uint64_t)v[i] + (odd ? FpConst::P(i) : 0u);
        v[i] = (uint32_t)cy;
        cy >>= 32;
      }
      for (int i = 0; i < NL; i++) v[i] = (v[i] >> 1) | ((i + 1 < NL ? v[i + 1] : (uint32_t)cy) << 31);
    }
    for (int j = 0; j < 16; j++) {
      const int w = (28 * j) / 32, s = (28 * j) % 32;
      const uint64_t q = (uint64_t)v[w] | ((uint64_t)(w + 1 < NL ? v[w + 1] : 0u) << 32);
      t.fold[k][(j + 14) % 16] = (int32_t)((q >> s) & (uint64_t)WM28);
    }
  }
  for (int j = 0; j < 16; j++) t.p[j] = p28(j);
  for (int l = 0; l < 8; l++) {
    t.pm[l][0] = l == 7 ? p28(15) : p28(2 * l + 1);
    t.pm[l][1] = l == 7 ? p28(0) : p28(2 * l + 2);
    t.pm[l][2] = l == 7 ? p28(1) : p28(2 * l + 3);
  }
  return t;
}

static __device__ const WarpTable W_TABLE = make_warp_table();

// -p^-1 mod 2^56
constexpr uint64_t w_np56() {
  const uint64_t p0 = (uint64_t)FpConst::P(0) | ((uint64_t)FpConst::P(1) << 32);
  uint64_t x = 1;
  for (int i = 0; i < 6; i++) x *= 2 - p0 * x;
  return (0 - x) & ((1ull << 56) - 1);
}

// Scratch of one warp, in 32-bit words: operand a, operand b (doubled; the
// group stride of 48 words keeps two groups' pair reads on disjoint banks)
// and the folded limbs t, for N products (1 for Fp, 3 for an Fp2 product).
template <class F>
struct WScratch;
template <>
struct WScratch<Fp> {
  static constexpr int N = 1, NT = 1;
};
template <>
struct WScratch<Fp2> {
  static constexpr int N = 3, NT = 2;
};
constexpr int W_A = 4 * 16, W_B = 4 * 48, W_T = 4 * 16;
constexpr int W_TABLE_WORDS = sizeof(WarpTable) / 4;
static_assert(W_TABLE_WORDS % 4 == 0, "scratch alignment");

template <class F>
constexpr int w_scratch_words() {
  return WScratch<F>::N * (W_A + W_B) + WScratch<F>::NT * W_T;
}
template <class F>
constexpr int w_smem_bytes(int warps) {
  return 4 * (W_TABLE_WORDS + warps * w_scratch_words<F>());
}

extern __shared__ __align__(16) int32_t w_smem[];

// Index of the warp in its block, through a shuffle: the compiler then knows
// branches on it as uniform and leaves out their reconvergence.
GM_DEVI int w_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
GM_DEVI int w_lane() { return (int)(threadIdx.x & 7u); }
GM_DEVI int w_group() { return (int)((threadIdx.x >> 3) & 3u); }
GM_DEVI const WarpTable &w_table() { return *reinterpret_cast<const WarpTable *>(w_smem); }
template <class F>
GM_DEVI int32_t *w_scratch() {
  return w_smem + W_TABLE_WORDS + (threadIdx.x >> 5) * w_scratch_words<F>();
}
// Copies the tables into shared memory; every thread of the block calls it.
GM_DEVI void w_setup() {
  const int32_t *src = reinterpret_cast<const int32_t *>(&W_TABLE);
  for (int i = threadIdx.x; i < W_TABLE_WORDS; i += blockDim.x) w_smem[i] = __ldg(src + i);
  __syncthreads();
}

struct wfp {
  int32_t l0, l1;
};
struct wfp2 {
  wfp c0, c1;
};

struct WCols {
  int64_t lo0, lo1, hi0, hi1;  // columns 2l, 2l+1 and 2l+16, 2l+17
};

// One carry pass: limbs of any int32 value -> [-8, 2^28 + 8], value unchanged.
GM_DEVI wfp w_carry(const wfp &v) {
  const int l = w_lane();
  const int32_t q0 = v.l0 >> 28, q1 = v.l1 >> 28;
  int32_t r = __shfl_up_sync(0xffffffffu, q1, 1, 8);
  if (l == 0) r = 0;
  return wfp{(v.l0 & WM28) + r, (l == 7 ? v.l1 : (v.l1 & WM28)) + q0};
}

// v - round(v / p) p for |v| < 20 p with |limbs| + 2^28 |v / p| < 2^31:
// |result| < 0.51 p, carried.  The quotient comes from the top limb alone
// (p >> 420 has 26 bits; the limbs below it move it by less than 2^-20).
GM_DEVI wfp w_reduce(const wfp &v) {
  constexpr int64_t C = (int64_t)(((uint64_t)1 << 40) / ((uint64_t)p28(15) + 1));  // 2^40 / (p >> 420), low by < 2^-25
  const int32_t top = __shfl_sync(0xffffffffu, v.l1, 7, 8);
  const int32_t q = (int32_t)(((int64_t)top * C + ((int64_t)1 << 39)) >> 40);
  const int2 p = reinterpret_cast<const int2 *>(w_table().p)[w_lane()];
  return w_carry(wfp{v.l0 - q * p.x, v.l1 - q * p.y});
}

GM_DEVI wfp w_add(const wfp &a, const wfp &b) { return wfp{a.l0 + b.l0, a.l1 + b.l1}; }
GM_DEVI wfp w_sub(const wfp &a, const wfp &b) { return wfp{a.l0 - b.l0, a.l1 - b.l1}; }

// a and b (this lane's limbs) to the group's slots
GM_DEVI void w_put(int32_t *sa, int32_t *sb, const wfp &a, const wfp &b) {
  const int l = w_lane(), g = w_group();
  reinterpret_cast<int2 *>(sa + g * 16)[l] = make_int2(a.l0, a.l1);
  int2 *pb = reinterpret_cast<int2 *>(sb + g * 48);
  pb[l] = make_int2(b.l0, b.l1);
  pb[l + 8] = make_int2(b.l0, b.l1);
}

// Columns of a * b from the group's slots (per group).
GM_DEVI WCols w_columns(const int32_t *sa, const int32_t *sb) {
  const int l = w_lane(), g = w_group();
  const int4 *pa = reinterpret_cast<const int4 *>(sa + g * 16);
  const int2 *pb = reinterpret_cast<const int2 *>(sb + g * 48) + 8 + l;
  int32_t a[16];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int4 v = pa[i];
    a[4 * i] = v.x;
    a[4 * i + 1] = v.y;
    a[4 * i + 2] = v.z;
    a[4 * i + 3] = v.w;
  }
  WCols r;
  int64_t c0 = 0, c1 = 0;
  int32_t bw = 0;  // odd limb of this lane's own pair: a_15 times it wraps into column 2l + 16
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int2 b = pb[-i];
    if (i == 0)
      bw = b.y;
    else
      c0 += (int64_t)a[2 * i - 1] * b.y;
    c0 += (int64_t)a[2 * i] * b.x;
    c1 += (int64_t)a[2 * i] * b.y;
    c1 += (int64_t)a[2 * i + 1] * b.x;
    if (i == l) {
      r.lo0 = c0;
      r.lo1 = c1;
    }
  }
  c0 += (int64_t)a[15] * bw;
  r.hi0 = c0 - r.lo0;
  r.hi1 = c1 - r.lo1;
  return r;
}

// Montgomery reduction of N column sets (|columns| < 2^62), per group.
template <int N>
GM_DEVI void w_redc(wfp (&out)[N], const WCols (&t)[N], int32_t *st) {
  const int l = w_lane(), g = w_group();
  const WarpTable &tab = w_table();
  int64_t f0[N], f1[N];
#pragma unroll
  for (int n = 0; n < N; n++) {
    const int32_t x0 = (int32_t)t[n].lo0 & WM28, y0 = (int32_t)(t[n].lo0 >> 28) & WM28;
    const int32_t x1 = (int32_t)t[n].lo1 & WM28, y1 = (int32_t)(t[n].lo1 >> 28) & WM28;
    const int32_t z0 = (int32_t)(t[n].lo0 >> 56), z1 = (int32_t)(t[n].lo1 >> 56);
    int32_t r0 = __shfl_up_sync(0xffffffffu, y1 + z0, 1, 8);
    int32_t r1 = __shfl_up_sync(0xffffffffu, z1, 1, 8);
    if (l == 0) r0 = r1 = 0;
    reinterpret_cast<int2 *>(st + n * W_T + g * 16)[l] = make_int2(x0 + r0, x1 + y0 + r1);
    f0[n] = l == 7 ? t[n].lo0 + r0 : t[n].hi0;
    f1[n] = l == 7 ? t[n].lo1 + r1 : t[n].hi1;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < W_FOLD; k += 2) {
    const int2 d0 = reinterpret_cast<const int2 *>(tab.fold[k])[l];
    const int2 d1 = reinterpret_cast<const int2 *>(tab.fold[k + 1])[l];
#pragma unroll
    for (int n = 0; n < N; n++) {
      const int2 tk = *reinterpret_cast<const int2 *>(st + n * W_T + g * 16 + k);
      f0[n] += (int64_t)tk.x * d0.x;
      f1[n] += (int64_t)tk.x * d0.y;
      f0[n] += (int64_t)tk.y * d1.x;
      f1[n] += (int64_t)tk.y * d1.y;
    }
  }
  const int4 pm = *reinterpret_cast<const int4 *>(tab.pm[l]);
#pragma unroll
  for (int n = 0; n < N; n++) {
    constexpr uint64_t NP = w_np56();
    const uint64_t m = ((uint64_t)f0[n] + ((uint64_t)f1[n] << 28)) * NP;  // lane 7's is the one used
    const int32_t m0 = __shfl_sync(0xffffffffu, (int32_t)(m & (uint64_t)WM28), 7, 8);
    const int32_t m1 = __shfl_sync(0xffffffffu, (int32_t)((m >> 28) & (uint64_t)WM28), 7, 8);
    const int64_t e = (int64_t)m1 * pm.x + (l == 7 ? t[n].hi0 : f0[n]);
    int64_t c0 = f0[n] + (int64_t)m0 * pm.y;
    int64_t c1 = f1[n] + (int64_t)m0 * pm.z + (int64_t)m1 * pm.y;
    // lane 7: c0, c1 are V's columns 0 and 1, now 0 mod 2^56; their carry goes to column 2 (lane 0), and the
    // lane's own result is column 14 (column 15 is 0)
    c1 += l == 7 ? c0 >> 28 : 0;
    c0 = l == 7 ? e : e + (int64_t)m0 * pm.y;
    const int32_t x0 = (int32_t)c0 & WM28, y0 = (int32_t)(c0 >> 28) & WM28, z0 = (int32_t)(c0 >> 56);
    const int32_t x1 = (int32_t)c1 & WM28, y1 = (int32_t)(c1 >> 28) & WM28, z1 = (int32_t)(c1 >> 56);
    const int32_t r0 = __shfl_sync(0xffffffffu, l == 7 ? y1 : y1 + z0, (l + 7) & 7, 8);
    const int32_t r1 = __shfl_sync(0xffffffffu, z1, (l + 7) & 7, 8);
    out[n] = w_carry(wfp{x0 + r0, l == 7 ? (int32_t)(c0 >> 28) + r1 : x1 + y0 + r1});
  }
}

// Element in memory (14 words) -> limbs of this lane: the three words that
// hold them, and the limbs cut out of these.
struct wwords {
  uint32_t w0, w1, w2;
};
GM_DEVI wwords w_fetch(const uint32_t *w) {
  const int j = (7 * w_lane()) >> 2;
  return wwords{w[j], w[j + 1], w[min(j + 2, NL - 1)]};
}
GM_DEVI wfp w_cut(const wwords &v) {
  const int s = (24 * w_lane()) & 31;
  const uint32_t lo = __funnelshift_r(v.w0, v.w1, s), hi = __funnelshift_r(v.w1, v.w2, s);
  return wfp{(int32_t)(lo & (uint32_t)WM28), (int32_t)(((lo >> 28) | (hi << 4)) & (uint32_t)WM28)};
}
GM_DEVI wfp w_load(const uint32_t *w) { return w_cut(w_fetch(w)); }

// Canonical value (per group; every lane of a group gets it) of |v| < 20 p.
// st: the group's t slot.
GM_DEVI fp_t w_canon(const wfp &v, int32_t *st) {
  const wfp r = w_reduce(v);
  const int l = w_lane(), g = w_group();
  __syncwarp();
  reinterpret_cast<int2 *>(st + g * 16)[l] = make_int2(r.l0, r.l1);
  __syncwarp();
  const int4 *p4 = reinterpret_cast<const int4 *>(st + g * 16);
  int32_t c = 0;
  uint64_t acc = 0;  // packed low bits
  int bits = 0, j = 0;
  fp_t o;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int4 v4 = p4[q];
    const int32_t x[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int32_t s = x[e] + p28(4 * q + e) + c;  // v + p > 0
      c = s >> 28;
      acc |= (uint64_t)(uint32_t)(s & WM28) << bits;
      bits += 28;
      if (bits >= 32) {
        o.v[j++] = (uint32_t)acc;
        acc >>= 32;
        bits -= 32;
      }
    }
  }
  cond_sub<false>(o.v);
  return o;
}

// v == 0 mod p for a value with |v| < 3 p, equal in the four groups.  v's
// lowest 28 bits decide except with probability 2^-25: a multiple j p of p
// has lowest bits j p mod 2^28.
GM_DEVI bool w_maybe_zero(const wfp &v) {
  constexpr uint32_t PI = 0u - FpConst::PINV;  // p^-1 mod 2^32
  const uint32_t j = (uint32_t)v.l0 * PI + 4u;
  return __shfl_sync(0xffffffffu, (j & (uint32_t)WM28) < 8u ? 1 : 0, 0) != 0;
}

// a^-1 R^2 for a Montgomery-form a = x R, i.e. x^-1 R; 0 -> 0.  Equal in the
// four groups.  Division steps of Bernstein and Yang ("Fast constant-time gcd
// computation and modular inversion", 2019) on f = p, g = a: 28 steps depend
// on the low 28 bits of f and g alone and multiply (f, g) by a matrix of
// entries up to 2^28 over 2^28, which every lane works out for itself; the
// same matrix, with an exact division by 2^28 modulo p, acts on (d, e), kept
// at d a = f R^2 and e a = g R^2 modulo p.  Groups 0 and 1 hold f and g and
// compute the next ones, groups 2 and 3 d and e.  1288 steps suffice for 446
// bits (their Theorem 11.2); the loop ends when g is 0, after about 36 rounds
// of 1050 cycles (20 us), a tenth of an exponentiation by p - 2.
static __device__ __noinline__ wfp w_inv_fp(wfp a) {
  const int l = w_lane(), grp = w_group();
  const int2 p = reinterpret_cast<const int2 *>(w_table().p)[l];
  constexpr int64_t C = (int64_t)(((uint64_t)1 << 40) / ((uint64_t)p28(15) + 1));  // as in w_reduce
  const int jw = (7 * l) >> 2;
  a = w_reduce(a);
  const wfp r2 = w_cut(wwords{FpConst::R2(jw), FpConst::R2(jw + 1), FpConst::R2(min(jw + 2, NL - 1))});
  wfp A = grp < 2 ? wfp{p.x, p.y} : wfp{0, 0};
  wfp B = grp < 2 ? a : r2;
  int32_t delta = 1;
#pragma unroll 1
  for (int it = 0; it < 47; it++) {
    if (__ballot_sync(0xffffffffu, grp < 2 && (B.l0 | B.l1) != 0) == 0) break;
    uint32_t f = (uint32_t)__shfl_sync(0xffffffffu, A.l0, 0), g = (uint32_t)__shfl_sync(0xffffffffu, B.l0, 0);
    int32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 4
    for (int s = 0; s < 28; s++) {
      const bool odd = g & 1u;
      const bool sw = odd && delta > 0;
      const uint32_t f1 = sw ? g : f, g1 = sw ? 0u - f : g;
      const int32_t u1 = sw ? q : u, v1 = sw ? r : v;
      const int32_t q1 = sw ? -u : q, r1 = sw ? -v : r;
      delta = (sw ? -delta : delta) + 1;
      f = f1;
      g = (g1 + (odd ? f1 : 0u)) >> 1;
      q = q1 + (odd ? u1 : 0);
      r = r1 + (odd ? v1 : 0);
      u = u1 << 1;
      v = v1 << 1;
    }
    const int32_t ca = (grp & 1) ? q : u, cb = (grp & 1) ? r : v;
    int64_t c0 = (int64_t)ca * A.l0 + (int64_t)cb * B.l0;
    int64_t c1 = (int64_t)ca * A.l1 + (int64_t)cb * B.l1;
    // m = 0 for f and g, whose lowest limb is divisible already
    const int32_t m = __shfl_sync(0xffffffffu, (int32_t)(((uint32_t)c0 * FpConst::PINV) & (uint32_t)WM28), 0, 8);
    c0 += (int64_t)m * p.x;
    c1 += (int64_t)m * p.y;
    const int32_t x0 = (int32_t)c0 & WM28, y0 = (int32_t)(c0 >> 28) & WM28, z0 = (int32_t)(c0 >> 56);
    const int32_t x1 = (int32_t)c1 & WM28, y1 = (int32_t)(c1 >> 28) & WM28, z1 = (int32_t)(c1 >> 56);
    int32_t r0 = __shfl_up_sync(0xffffffffu, y1 + z0, 1, 8), r1 = __shfl_up_sync(0xffffffffu, z1, 1, 8);
    if (l == 0) r0 = r1 = 0;
    const int32_t up = __shfl_down_sync(0xffffffffu, x0 + r0, 1, 8);  // limb 2l + 2
    wfp n{x1 + y0 + r1, l == 7 ? (int32_t)(c1 >> 28) + z0 : up};      // one limb down
    const int32_t top = __shfl_sync(0xffffffffu, n.l1, 7, 8);
    const int32_t qd = grp < 2 ? 0 : (int32_t)(((int64_t)top * C + ((int64_t)1 << 39)) >> 40);
    n = w_carry(wfp{n.l0 - qd * p.x, n.l1 - qd * p.y});
    const wfp o{__shfl_xor_sync(0xffffffffu, n.l0, 8), __shfl_xor_sync(0xffffffffu, n.l1, 8)};
    A = (grp & 1) ? o : n;
    B = (grp & 1) ? n : o;
  }
  const bool neg = ((uint32_t)__shfl_sync(0xffffffffu, A.l0, 0) & (uint32_t)WM28) != 1u;  // f = 1 or -1
  const wfp d{__shfl_sync(0xffffffffu, A.l0, 16 + l), __shfl_sync(0xffffffffu, A.l1, 16 + l)};
  return neg ? wfp{-d.l0, -d.l1} : d;
}

// ---------------------------------------------------------------------------
// Field policies
// ---------------------------------------------------------------------------
template <class F>
struct WF;

// Inline: a call's argument moves cost more than its 350 instructions (B200,
// one warp: doubling 2750 against 3100 cycles, addition 3530 against 3900).
static __device__ __forceinline__ wfp w_mul_fp(wfp a, wfp b) {
  int32_t *s = w_scratch<Fp>();
  w_put(s, s + W_A, a, b);
  __syncwarp();
  const WCols t[1] = {w_columns(s, s + W_A)};
  wfp r[1];
  w_redc<1>(r, t, s + W_A + W_B);
  return r[0];
}

template <>
struct WF<Fp> {
  using E = wfp;
  using T = fp_t;
  static constexpr int WORDS = 14;
  GM_DEVI static E zero() { return wfp{0, 0}; }
  GM_DEVI static E add(const E &a, const E &b) { return w_add(a, b); }
  GM_DEVI static E sub(const E &a, const E &b) { return w_sub(a, b); }
  GM_DEVI static E reduce(const E &a) { return w_reduce(a); }
  // 2 a as a factor (limbs below 2^29 + 16 are)
  GM_DEVI static E twice(const E &a) { return w_add(a, a); }
  // difference as a factor of values below 2 p
  GM_DEVI static E diff(const E &a, const E &b) { return w_sub(a, b); }
  GM_DEVI static E mul(const E &a, const E &b) { return w_mul_fp(a, b); }
  GM_DEVI static E inv(const E &a) { return w_inv_fp(a); }
  using Raw = wwords;
  GM_DEVI static Raw fetch(const uint32_t *w) { return w_fetch(w); }
  GM_DEVI static E cut(const Raw &v) { return w_cut(v); }
  GM_DEVI static E load(const T *p) { return w_load(reinterpret_cast<const uint32_t *>(p)); }
  GM_DEVI static E load_words(const uint32_t *w) { return w_load(w); }
  GM_DEVI static E from(const E &r, int g) {
    const int src = g * 8 + w_lane();
    return wfp{__shfl_sync(0xffffffffu, r.l0, src), __shfl_sync(0xffffffffu, r.l1, src)};
  }
  GM_DEVI static E pick(int g, const E &a0, const E &a1, const E &a2, const E &a3) {
    const E lo = (g & 1) ? a1 : a0, hi = (g & 1) ? a3 : a2;
    return (g & 2) ? hi : lo;
  }
  GM_DEVI static T canon(const E &v) { return w_canon(v, w_scratch<Fp>() + W_A + W_B); }
  GM_DEVI static bool is_zero(const E &v) {
    if (!w_maybe_zero(v)) return false;
    return Fp::is_zero_raw(canon(v));
  }
  GM_DEVI static bool raw_zero(const E &v) { return __ballot_sync(0xffffffffu, (v.l0 | v.l1) != 0) == 0; }
  // limbs to and from shared memory
  GM_DEVI static void put(int32_t *s, const E &v) { reinterpret_cast<int2 *>(s)[w_lane()] = make_int2(v.l0, v.l1); }
  GM_DEVI static E get(const int32_t *s) {
    const int2 v = reinterpret_cast<const int2 *>(s)[w_lane()];
    return wfp{v.x, v.y};
  }
  static constexpr int LW = 16;  // words of an element in shared memory
  GM_DEVI static E one() {
    const int j = (7 * w_lane()) >> 2;
    return w_cut(wwords{FpConst::ONE(j), FpConst::ONE(j + 1), FpConst::ONE(min(j + 2, NL - 1))});
  }
};

// Fp2 = Fp[i]/(i^2 + 1): Karatsuba on the columns, one reduction per
// coefficient.  Results are reduced to |c| < 0.51 p: a difference of two
// products would otherwise grow from formula to formula.  Out of line: inline
// copies outgrow the instruction cache (addition 8040 against 7530 cycles).
static __device__ __noinline__ wfp2 w_mul_fp2(wfp2 a, wfp2 b) {
  int32_t *s = w_scratch<Fp2>();
  constexpr int S = W_A + W_B;
  w_put(s, s + W_A, a.c0, b.c0);
  w_put(s + S, s + S + W_A, a.c1, b.c1);
  w_put(s + 2 * S, s + 2 * S + W_A, w_add(a.c0, a.c1), w_add(b.c0, b.c1));
  __syncwarp();
  WCols t[2];
  t[0] = w_columns(s, s + W_A);
  const WCols t1 = w_columns(s + S, s + S + W_A);
  t[1] = w_columns(s + 2 * S, s + 2 * S + W_A);
  t[1].lo0 -= t[0].lo0 + t1.lo0;
  t[1].lo1 -= t[0].lo1 + t1.lo1;
  t[1].hi0 -= t[0].hi0 + t1.hi0;
  t[1].hi1 -= t[0].hi1 + t1.hi1;
  t[0].lo0 -= t1.lo0;
  t[0].lo1 -= t1.lo1;
  t[0].hi0 -= t1.hi0;
  t[0].hi1 -= t1.hi1;
  wfp r[2];
  w_redc<2>(r, t, s + 3 * S);
  return wfp2{w_reduce(r[0]), w_reduce(r[1])};
}

template <>
struct WF<Fp2> {
  using E = wfp2;
  using T = fp2_t;
  using B = WF<Fp>;
  static constexpr int WORDS = 28;
  GM_DEVI static E zero() { return wfp2{B::zero(), B::zero()}; }
  GM_DEVI static E add(const E &a, const E &b) { return wfp2{w_add(a.c0, b.c0), w_add(a.c1, b.c1)}; }
  GM_DEVI static E sub(const E &a, const E &b) { return wfp2{w_sub(a.c0, b.c0), w_sub(a.c1, b.c1)}; }
  GM_DEVI static E reduce(const E &a) { return wfp2{w_reduce(a.c0), w_reduce(a.c1)}; }
  // carried: the Karatsuba sum of a factor doubles its limbs
  GM_DEVI static E twice(const E &a) { return wfp2{w_carry(w_add(a.c0, a.c0)), w_carry(w_add(a.c1, a.c1))}; }
  GM_DEVI static E diff(const E &a, const E &b) { return sub(a, b); }
  GM_DEVI static E mul(const E &a, const E &b) { return w_mul_fp2(a, b); }
  // conj(a) / (a conj(a))
  GM_DEVI static E inv(const E &a) {
    const E c{a.c0, w_sub(wfp{0, 0}, a.c1)};
    return mul(c, wfp2{w_inv_fp(mul(a, c).c0), wfp{0, 0}});
  }
  struct Raw {
    wwords c0, c1;
  };
  GM_DEVI static Raw fetch(const uint32_t *w) { return Raw{w_fetch(w), w_fetch(w + NL)}; }
  GM_DEVI static E cut(const Raw &v) { return wfp2{w_cut(v.c0), w_cut(v.c1)}; }
  GM_DEVI static E load(const T *p) { return wfp2{B::load(&p->c0), B::load(&p->c1)}; }
  GM_DEVI static E load_words(const uint32_t *w) { return wfp2{w_load(w), w_load(w + 14)}; }
  GM_DEVI static E from(const E &r, int g) { return wfp2{B::from(r.c0, g), B::from(r.c1, g)}; }
  GM_DEVI static E pick(int g, const E &a0, const E &a1, const E &a2, const E &a3) {
    return wfp2{B::pick(g, a0.c0, a1.c0, a2.c0, a3.c0), B::pick(g, a0.c1, a1.c1, a2.c1, a3.c1)};
  }
  GM_DEVI static T canon(const E &v) {
    int32_t *st = w_scratch<Fp2>() + 3 * (W_A + W_B);
    return fp2_t{w_canon(v.c0, st), w_canon(v.c1, st)};
  }
  GM_DEVI static bool is_zero(const E &v) {
    if (!w_maybe_zero(v.c0) || !w_maybe_zero(v.c1)) return false;
    const T c = canon(v);
    return Fp::is_zero_raw(c.c0) && Fp::is_zero_raw(c.c1);
  }
  GM_DEVI static bool raw_zero(const E &v) { return B::raw_zero(v.c0) && B::raw_zero(v.c1); }
  GM_DEVI static void put(int32_t *s, const E &v) {
    B::put(s, v.c0);
    B::put(s + 16, v.c1);
  }
  GM_DEVI static E get(const int32_t *s) { return wfp2{B::get(s), B::get(s + 16)}; }
  static constexpr int LW = 32;
  GM_DEVI static E one() { return wfp2{B::one(), B::zero()}; }
};

}  // namespace gm
