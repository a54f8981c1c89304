// XYZZ point arithmetic on a warp (warp_field.cuh): each of the four groups of
// eight lanes computes one field product of a formula level, so an addition
// (add-2008-s, 12M + 2S) has a serial depth of 4 products, a mixed addition
// (madd-2008-s) of 4 and a doubling (dbl-2008-s-1) of 3.
//
// Contract: all 32 lanes call together; points are equal in the four groups;
// every branch depends on warp-uniform values only.
//
// Value ranges (in units of p).  Coordinates enter as canonical loads, in
// [0, 1), or as results: X and Y reduced, |.| < 0.51, ZZ and ZZZ within 2.
// Fp products stay within (-1, 2), so the differences P and R stay within 3
// and their squares within 3.2; X3 and Y3 stay within 7 and are reduced.  Fp2
// products come reduced.  M = 3 X^2 is reduced before it is squared.
#pragma once
#include "warp_field.cuh"
#include "xyzz.cuh"

namespace gm {

template <class F>
struct wpt {
  typename WF<F>::E X, Y, ZZ, ZZZ;
  bool inf;
};

template <class F>
GM_DEVI wpt<F> w_inf() {
  using W = WF<F>;
  return wpt<F>{W::zero(), W::zero(), W::zero(), W::zero(), true};
}

// p = 2p.  Levels: {V = U^2, xx = X^2} -> {W = U V, S = X V, M^2, ZZ V}
// -> {M (S - X3), W Y, ZZZ W}.
template <class F>
__device__ __noinline__ wpt<F> w_dbl(wpt<F> p) {
  using W = WF<F>;
  using E = typename W::E;
  if (p.inf) return p;
  if (W::is_zero(p.Y)) return w_inf<F>();  // 2-torsion
  const int g = w_group();
  const E U = W::twice(p.Y);
  E r = W::pick(g, U, p.X, U, p.X);
  r = W::mul(r, r);
  const E V = W::from(r, 0), xx = W::from(r, 1);
  const E M = W::reduce(W::add(W::add(xx, xx), xx));
  r = W::mul(W::pick(g, U, p.X, M, p.ZZ), W::pick(g, V, V, M, V));
  const E Wv = W::from(r, 0), S = W::from(r, 1), MM = W::from(r, 2);
  p.ZZ = W::from(r, 3);
  p.X = W::reduce(W::sub(MM, W::add(S, S)));
  r = W::mul(W::pick(g, M, Wv, Wv, Wv), W::pick(g, W::diff(S, p.X), p.Y, p.ZZZ, p.ZZZ));
  p.Y = W::reduce(W::sub(W::from(r, 0), W::from(r, 1)));
  p.ZZZ = W::from(r, 2);
  return p;
}

// Common end of both additions: from P, R, the first operand's U1, S1 and
// the products' second level.
template <class F>
GM_DEVI void w_add_tail(wpt<F> &acc, const typename WF<F>::E &P, const typename WF<F>::E &R,
                        const typename WF<F>::E &U1, const typename WF<F>::E &S1, const typename WF<F>::E &PP,
                        const typename WF<F>::E &RR, const typename WF<F>::E &ZZ, const typename WF<F>::E &ZZZ) {
  using W = WF<F>;
  using E = typename W::E;
  const int g = w_group();
  E r = W::mul(W::pick(g, P, U1, ZZ, ZZ), PP);
  const E PPP = W::from(r, 0), Q = W::from(r, 1);
  acc.ZZ = W::from(r, 2);
  acc.X = W::reduce(W::sub(W::sub(RR, PPP), W::add(Q, Q)));
  r = W::mul(W::pick(g, R, S1, ZZZ, ZZZ), W::pick(g, W::diff(Q, acc.X), PPP, PPP, PPP));
  acc.Y = W::reduce(W::sub(W::from(r, 0), W::from(r, 1)));
  acc.ZZZ = W::from(r, 2);
}

// acc + o, same exceptional cases as xyzz_add: an infinite operand, P == Q
// (doubling) and P == -Q (infinity).  Levels: {U1, U2, S1, S2} -> {P^2, R^2,
// ZZ1 ZZ2, ZZZ1 ZZZ2} -> {P PP, U1 PP, ZZ12 PP} -> {R (Q - X3), S1 PPP, ZZZ12 PPP}.
template <class F>
__device__ __noinline__ wpt<F> w_addp(wpt<F> acc, wpt<F> o) {
  using W = WF<F>;
  using E = typename W::E;
  if (o.inf) return acc;
  if (acc.inf) return o;
  const int g = w_group();
  E r = W::mul(W::pick(g, acc.X, o.X, acc.Y, o.Y), W::pick(g, o.ZZ, acc.ZZ, o.ZZZ, acc.ZZZ));
  const E U1 = W::from(r, 0), S1 = W::from(r, 2);
  const E P = W::diff(W::from(r, 1), U1);
  const E R = W::diff(W::from(r, 3), S1);
  if (W::is_zero(P)) {
    if (W::is_zero(R)) return w_dbl<F>(acc);
    return w_inf<F>();
  }
  r = W::mul(W::pick(g, P, R, acc.ZZ, acc.ZZZ), W::pick(g, P, R, o.ZZ, o.ZZZ));
  w_add_tail<F>(acc, P, R, U1, S1, W::from(r, 0), W::from(r, 1), W::from(r, 2), W::from(r, 3));
  return acc;
}

// acc + (x, y), an affine point that is not at infinity.
template <class F>
__device__ __noinline__ wpt<F> w_madd(wpt<F> acc, typename WF<F>::E x, typename WF<F>::E y) {
  using W = WF<F>;
  using E = typename W::E;
  if (acc.inf) return wpt<F>{x, y, W::one(), W::one(), false};
  const int g = w_group();
  E r = W::mul(W::pick(g, x, y, x, y), W::pick(g, acc.ZZ, acc.ZZZ, acc.ZZ, acc.ZZZ));
  const E P = W::diff(W::from(r, 0), acc.X);
  const E R = W::diff(W::from(r, 1), acc.Y);
  if (W::is_zero(P)) {
    if (W::is_zero(R)) return w_dbl<F>(acc);
    return w_inf<F>();
  }
  r = W::pick(g, P, R, P, R);
  r = W::mul(r, r);
  w_add_tail<F>(acc, P, R, acc.X, acc.Y, W::from(r, 0), W::from(r, 1), acc.ZZ, acc.ZZZ);
  return acc;
}

// k * p for a small non-negative integer k (MSB-first double-and-add)
template <class F>
GM_DEVI wpt<F> w_mul_small(const wpt<F> &p, uint32_t k) {
  wpt<F> r = w_inf<F>();
  if (k == 0 || p.inf) return r;
  r = p;
  for (int b = 30 - __clz(k); b >= 0; b--) {
    r = w_dbl<F>(r);
    if ((k >> b) & 1u) r = w_addp<F>(r, p);
  }
  return r;
}

// Points in device memory (canonical; infinity is ZZ = 0)
template <class F>
GM_DEVI wpt<F> w_load_pt(const xyzz_t<F> *p) {
  using W = WF<F>;
  wpt<F> r{W::load(&p->X), W::load(&p->Y), W::load(&p->ZZ), W::load(&p->ZZZ), false};
  r.inf = W::raw_zero(r.ZZ);
  return r;
}
// Each group makes one coordinate canonical and writes it.
template <class F>
GM_DEVI void w_store_pt(xyzz_t<F> *p, const wpt<F> &v) {
  using W = WF<F>;
  const int g = w_group();
  const wpt<F> z = v.inf ? w_inf<F>() : v;
  const typename F::T c = W::canon(W::pick(g, z.X, z.Y, z.ZZ, z.ZZZ));
  if (w_lane() == 0) reinterpret_cast<typename F::T *>(p)[g] = c;
}

// Points in shared memory, in limbs: W_PT words each
template <class F>
constexpr int w_pt_words() {
  return 4 * WF<F>::LW + 4;
}
template <class F>
GM_DEVI void w_put_pt(int32_t *s, const wpt<F> &v) {
  using W = WF<F>;
  const int g = w_group();
  W::put(s + g * W::LW, W::pick(g, v.X, v.Y, v.ZZ, v.ZZZ));
  if ((threadIdx.x & 31u) == 0) s[4 * W::LW] = v.inf ? 1 : 0;
}
template <class F>
GM_DEVI wpt<F> w_get_pt(const int32_t *s) {
  using W = WF<F>;
  return wpt<F>{W::get(s), W::get(s + W::LW), W::get(s + 2 * W::LW), W::get(s + 3 * W::LW), s[4 * W::LW] != 0};
}

// dynamic shared memory of a block that also exchanges one point per warp
template <class F>
constexpr int w_sum_smem(int warps) {
  return w_smem_bytes<F>(warps) + 4 * warps * w_pt_words<F>();
}

// Sum of the points of a block's `warps` warps (a power of two) in warp 0;
// s: warps * w_pt_words<F>() words.  Every warp of the block calls it.
template <class F>
GM_DEVI wpt<F> w_block_sum(wpt<F> v, int warps, int32_t *s) {
  const int w = w_warp();
  for (int h = warps >> 1; h >= 1; h >>= 1) {
    if (w >= h && w < 2 * h) w_put_pt<F>(s + (w - h) * w_pt_words<F>(), v);
    __syncthreads();
    if (w < h) v = w_addp<F>(v, w_get_pt<F>(s + w * w_pt_words<F>()));
    __syncthreads();
  }
  return v;
}

}  // namespace gm
