// Bucket reduction, long-run fix-up and window combination for the MSM
// pipelines (single and batched).
//
// Bucket reduction.  Per window (group g of G) with B buckets V_0..V_{B-1}:
//     S_g = sum_j (j + 1) V_j.
// Level 0 cuts the buckets into segments of L0 and computes in one thread per
// segment, by a running sum from the top,
//     T_s = sum_r (r + 1) V_{s L0 + r},   A_s = sum_r V_{s L0 + r},
// two additions per bucket and nothing else.  Then
//     S_g = sum_s T_s + L0 * sum_s s A_s.
// Level 1 cuts the A_s into segments of L1; a warp per segment s' computes  D = sum_r r A_{s' L1 + r},  A' = sum_r A_{s' L1 + r}  and
//     E_{s'} = L0 * (D + (s' L1) A')          (double-and-add, then doublings)
// so that  sum_s s A_s = sum_{s'} (D + s' L1 A')  and
//     S_g = sum_s T_s + sum_{s'} E_{s'}.
// Block sums add the nseg0 + nseg1 values of every group.  Level 0 holds
// nearly all the work; the few, serial additions of level 1 and the sums run
// on warps (xyzz_warp.cuh) to cut their latency.  B200, against four lanes of
// one product each: G1 1024 points 0.92 -> 0.07 ms, G1 2^20 2.01 -> 1.56 ms,
// G2 2^18 3.94 -> 2.87 ms for the whole reduction.  This replaces the reference's per-block
// partial buckets and per-window host combine (src/curve.cu:1557-1654,
// :2060-2179) with work that stays on the device.
#pragma once
#include "msm_kernels.cuh"
#include "xyzz_chain.cuh"

namespace gm {

constexpr int W_THREADS = 128;    // block of the kernels with one warp per work item
constexpr int SUM_WARPS = 8;      // warps of a block sum
constexpr int COMBINE_WARPS = 8;  // groups of windows of a window combination, a warp each, beside the chain's warps
template <class F>
constexpr int COMBINE_THREADS = 32 * (COMBINE_WARPS + Chain<F>::WARPS);
constexpr int W_FILL = 16;        // warps per SM that keep its schedulers busy with dependent point operations
constexpr int ACC_WARP_MIN = 4;    // entries of a slice on a warp, at least
constexpr int ACC_WARP_MAX = 16;   // and at most; beyond four times W_FILL warps per SM of these, threads take the slices
constexpr int ACC_THREAD_MIN = 16;  // entries of a slice on a thread, at least
constexpr int RED_THREAD_MIN = 3;  // level 0 goes to threads above this many buckets per thread of a wave

// ---------------------------------------------------------------------------
// Bucket accumulation with one warp per slice, for MSMs with few entries.
// The slices, partials and outputs are those of k_accumulate.  A mixed
// addition is a chain of 10 products in one thread, 14 us, and 1.8 us in a
// warp (G1, B200), but it takes the multiplier of 12 thread additions; so a
// warp takes the slice while the slices of at least ACC_WARP_MIN entries fit
// the GPU's schedulers a few times over (acc_slices has the rule).
// ---------------------------------------------------------------------------
template <class F>
__global__ void __launch_bounds__(W_THREADS) k_accumulate_warp(
    const uint4 *__restrict__ bases, const uint32_t *__restrict__ entries, const uint32_t *__restrict__ offsets,
    int64_t K, int64_t nslices, xyzz_t<F> *__restrict__ buckets, xyzz_t<F> *__restrict__ part_head,
    xyzz_t<F> *__restrict__ part_tail, int32_t *__restrict__ head_key, int32_t *__restrict__ tail_key) {
  using W = WF<F>;
  using E = typename W::E;
  w_setup();
  grid_wait(bases, entries, offsets);
  grid_release();
  const int64_t t = (int64_t)blockIdx.x * (W_THREADS / 32) + w_warp();
  if (t >= nslices) return;
  const uint32_t M = __ldg(offsets + K);
  const uint64_t chunk64 = ((uint64_t)M + nslices - 1) / nslices;
  const uint32_t chunk = chunk64 > 0 ? (uint32_t)chunk64 : 1u;
  const uint64_t start64 = (uint64_t)t * chunk;
  int32_t hk = -1, tk = -1;
  if (start64 < M) {
    const uint32_t end = (uint32_t)(start64 + chunk < M ? start64 + chunk : M);
    uint32_t pos = (uint32_t)start64;
    int64_t k = bucket_of(offsets, K, pos);
    uint32_t bend = __ldg(offsets + k + 1);
    bool owns = __ldg(offsets + k) == pos;
    wpt<F> acc = w_inf<F>();
    uint32_t e = __ldg(entries + pos);
    const uint32_t *rec = reinterpret_cast<const uint32_t *>(bases + (size_t)(e >> 1) * Rec<F>::U4);
    typename W::Raw rx = W::fetch(rec), ry = W::fetch(rec + F::LIMBS);
    while (true) {
      const E x = W::cut(rx);
      E y = W::cut(ry);
      if (e & 1u) y = W::sub(W::zero(), y);
      if (pos + 1 < end) {  // the next base, on its way during this addition
        e = __ldg(entries + pos + 1);
        rec = reinterpret_cast<const uint32_t *>(bases + (size_t)(e >> 1) * Rec<F>::U4);
        rx = W::fetch(rec);
        ry = W::fetch(rec + F::LIMBS);
      }
      // packed records of the point at infinity hold x = y = 0
      if (!(W::raw_zero(x) && W::raw_zero(y))) acc = w_madd<F>(acc, x, y);
      pos++;
      if (pos == bend || pos == end) {
        if (!owns) {
          w_store_pt<F>(part_head + t, acc);
          hk = (int32_t)k;
        } else if (pos == bend) {
          w_store_pt<F>(buckets + k, acc);
        } else {
          w_store_pt<F>(part_tail + t, acc);
          tk = (int32_t)k;
        }
        if (pos == end) break;
        k = seek_bucket(offsets, k + 1, K, pos);
        bend = __ldg(offsets + k + 1);
        owns = true;
        acc = w_inf<F>();
      }
    }
  }
  if ((threadIdx.x & 31u) == 0) {
    head_key[t] = hk;
    tail_key[t] = tk;
  }
}

// Level 0: segments (group, s) in a grid-stride loop.  The host picks L0 so
// that all segments fit in one resident wave when it can (no partial second
// wave doubling the serial time).  X has M values per group; T_s goes to
// X[g*M + s], A_s to A0[g*nseg0 + s].  Empty buckets (equal offsets) are not
// read; an empty segment costs two stores.
template <class F>
__global__ void __launch_bounds__(128) k_red_level0(const xyzz_t<F> *__restrict__ buckets,
                                                       const uint32_t *__restrict__ offsets, int64_t G, int B, int L0,
                                                       int nseg0, xyzz_t<F> *__restrict__ X, int M,
                                                       xyzz_t<F> *__restrict__ A0) {
  using FA = typename OutOfLine<F>::type;
  const int64_t total = G * nseg0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int64_t g = t / nseg0;
    const int s = (int)(t % nseg0);
    const int64_t kb = g * B;
    xyzz_t<FA> acc, ws;
    xyzz_set_inf(acc);
    xyzz_set_inf(ws);
    const int j0 = s * L0, j1 = min(B, j0 + L0);
    if (__ldg(offsets + kb + j0) != __ldg(offsets + kb + j1)) {  // any entries in the segment
      for (int j = j1 - 1; j >= j0; j--) {
        if constexpr (sizeof(typename F::T) == sizeof(fp_t)) {
          if (__ldg(offsets + kb + j + 1) != __ldg(offsets + kb + j)) xyzz_add<FA>(acc, as_xyzz<FA>(buckets[kb + j]));
          xyzz_add<FA>(ws, acc);
        } else {
          // Fp2: the addition out of line keeps the loop within the register file
          if (__ldg(offsets + kb + j + 1) != __ldg(offsets + kb + j))
            xyzz_add_cold<FA>(acc, as_xyzz<FA>(buckets[kb + j]));
          xyzz_add_cold<FA>(ws, acc);
        }
      }
    }
    X[g * M + s] = as_xyzz<F>(ws);
    A0[g * nseg0 + s] = as_xyzz<F>(acc);
  }
}

// Level 0 on warps (warp_field.cuh): one warp per segment.  A segment's two
// additions per bucket are one serial chain, 40 us per bucket in one thread
// and 2.6 us in a warp (G1), so warps take over wherever the segments do not
// fill the GPU with threads (RedLayout::plan has the rule).
template <class F>
__global__ void __launch_bounds__(W_THREADS) k_red_level0_warp(const xyzz_t<F> *__restrict__ buckets,
                                                               const uint32_t *__restrict__ offsets, int64_t G, int B,
                                                               int L0, int nseg0, xyzz_t<F> *__restrict__ X, int M,
                                                               xyzz_t<F> *__restrict__ A0) {
  w_setup();
  grid_wait(buckets, offsets);
  grid_release();
  const int64_t t = (int64_t)blockIdx.x * (W_THREADS / 32) + w_warp();
  if (t >= G * nseg0) return;
  const int64_t g = t / nseg0;
  const int s = (int)(t % nseg0);
  const int64_t kb = g * B;
  wpt<F> acc = w_inf<F>(), ws = w_inf<F>();
  const int j0 = s * L0, j1 = min(B, j0 + L0);
  for (int j = j1 - 1; j >= j0; j--) {
    if (__ldg(offsets + kb + j + 1) != __ldg(offsets + kb + j)) acc = w_addp<F>(acc, w_load_pt<F>(buckets + kb + j));
    ws = w_addp<F>(ws, acc);
  }
  w_store_pt<F>(X + g * M + s, ws);
  w_store_pt<F>(A0 + g * nseg0 + s, acc);
}

// Level 1: one warp per (group, segment s').  Writes E_{s'} to X[g*M + nseg0 + s'].
template <class F>
__global__ void __launch_bounds__(W_THREADS) k_red_level1(const xyzz_t<F> *__restrict__ A0, int64_t G, int nseg0,
                                                          int L1, int nseg1, int L0, xyzz_t<F> *__restrict__ X, int M) {
  w_setup();
  grid_wait(A0);
  grid_release();
  const int64_t t = (int64_t)blockIdx.x * (W_THREADS / 32) + w_warp();
  if (t >= G * nseg1) return;
  const int64_t g = t / nseg1;
  const int s = (int)(t % nseg1);
  const int r0 = s * L1, r1 = min(nseg0, r0 + L1);
  wpt<F> acc = w_inf<F>(), ws = w_inf<F>();
  for (int r = r1 - 1; r >= r0; r--) {
    acc = w_addp<F>(acc, w_load_pt<F>(A0 + g * nseg0 + r));
    if (r > r0) ws = w_addp<F>(ws, acc);
  }
  // ws = sum (r - r0) A_r; add (s L1) * acc, then scale by L0
  ws = w_addp<F>(ws, w_mul_small<F>(acc, (uint32_t)r0));
  w_store_pt<F>(X + g * M + nseg0 + s, w_mul_small<F>(ws, (uint32_t)L0));
}

// out[g*nout + i] = sum of in[g*N + j], j in [i*chunk, (i+1)*chunk): one block
// of SUM_WARPS warps per output, strided sums and a tree in shared memory.
template <class F>
__global__ void __launch_bounds__(32 * SUM_WARPS) k_red_sum(const xyzz_t<F> *__restrict__ in, int N, int chunk,
                                                            int nout, xyzz_t<F> *__restrict__ out) {
  w_setup();
  grid_wait(in);
  grid_release();
  const int64_t g = blockIdx.x / nout;
  const int i = (int)(blockIdx.x % nout);
  const int j1 = min(N, (i + 1) * chunk);
  wpt<F> acc = w_inf<F>();
  for (int j = i * chunk + w_warp(); j < j1; j += SUM_WARPS) acc = w_addp<F>(acc, w_load_pt<F>(in + g * N + j));
  acc = w_block_sum<F>(acc, SUM_WARPS, w_smem + w_smem_bytes<F>(SUM_WARPS) / 4);
  if (threadIdx.x < 32) w_store_pt<F>(out + blockIdx.x, acc);
}

// ---------------------------------------------------------------------------
// Fix-up of buckets that straddle accumulation slices.  Slice t0 holds the
// tail piece of bucket k (part_tail[t0]); slices t0+1..t1 hold head pieces
// (part_head).  Runs of at most FIX_SHORT heads are folded serially by the
// owner of the tail; longer runs (a bucket much larger than a slice, e.g. all
// the scalars equal to 1) are queued and folded by k_fixup_long, one block of
// SUM_WARPS warps per run with a shared-memory tree.
// ---------------------------------------------------------------------------
constexpr int FIX_SHORT = 8;
constexpr int FIX_LONG_BLOCKS = 64;

// long_q: [0] = count, then bucket keys
template <class F>
__global__ void __launch_bounds__(W_THREADS) k_fixup_split(const uint32_t *__restrict__ offsets, int64_t K,
                                                           int64_t nslices, xyzz_t<F> *__restrict__ buckets,
                                                           const xyzz_t<F> *__restrict__ part_head,
                                                           const xyzz_t<F> *__restrict__ part_tail,
                                                           const int32_t *__restrict__ head_key,
                                                           const int32_t *__restrict__ tail_key,
                                                           uint32_t *__restrict__ err, int32_t *__restrict__ long_q,
                                                           int64_t long_cap) {
  w_setup();
  grid_wait(offsets, part_head, part_tail, head_key, tail_key);
  grid_release();
  const int64_t t = (int64_t)blockIdx.x * (W_THREADS / 32) + w_warp();
  if (t >= nslices) return;
  const int32_t k = __ldg(tail_key + t);
  if (k < 0) return;
  const uint32_t M = __ldg(offsets + K);
  const uint64_t chunk64 = ((uint64_t)M + nslices - 1) / nslices;
  const uint64_t chunk = chunk64 > 0 ? chunk64 : 1u;
  const uint64_t bend = __ldg(offsets + k + 1);
  const int64_t t1 = (int64_t)((bend - 1) / chunk);  // slice holding the bucket's last entry
  const bool lead = (threadIdx.x & 31u) == 0;
  if (t1 - t > FIX_SHORT) {
    if (lead) {
      const int32_t slot = atomicAdd(long_q, 1);
      if (slot < long_cap)
        long_q[1 + slot] = k;
      else
        atomicOr(err, 2u);
    }
    return;
  }
  wpt<F> acc = w_load_pt<F>(part_tail + t);
  for (int64_t t2 = t + 1; t2 <= t1 && t2 < nslices; t2++) {
    if (__ldg(head_key + t2) != k) {  // cannot happen for a consistent slicing
      if (lead) atomicOr(err, 1u);
      break;
    }
    acc = w_addp<F>(acc, w_load_pt<F>(part_head + t2));
  }
  w_store_pt<F>(buckets + k, acc);
}

template <class F>
__global__ void __launch_bounds__(32 * SUM_WARPS) k_fixup_long(const uint32_t *__restrict__ offsets, int64_t K,
                                                               int64_t nslices, xyzz_t<F> *__restrict__ buckets,
                                                               const xyzz_t<F> *__restrict__ part_head,
                                                               const xyzz_t<F> *__restrict__ part_tail,
                                                               const int32_t *__restrict__ head_key,
                                                               uint32_t *__restrict__ err,
                                                               const int32_t *__restrict__ long_q, int64_t long_cap) {
  w_setup();
  grid_wait(offsets, part_head, part_tail, head_key, long_q);
  grid_release();
  const int64_t n_long = min((int64_t)long_q[0], long_cap);
  if ((int64_t)blockIdx.x >= n_long) return;
  const int w = w_warp();
  const uint32_t M = __ldg(offsets + K);
  const uint64_t chunk64 = ((uint64_t)M + nslices - 1) / nslices;
  const uint64_t chunk = chunk64 > 0 ? chunk64 : 1u;
  for (int64_t item = blockIdx.x; item < n_long; item += gridDim.x) {
    const int32_t k = long_q[1 + item];
    const int64_t t0 = (int64_t)(__ldg(offsets + k) / chunk);
    const int64_t t1 = min((int64_t)((__ldg(offsets + k + 1) - 1) / chunk), nslices - 1);
    // warp w folds run positions w, w + SUM_WARPS, ... (position 0 is the tail piece)
    wpt<F> acc = w_inf<F>();
    for (int64_t p = w; p <= t1 - t0; p += SUM_WARPS) {
      const int64_t ts = t0 + p;
      if (p == 0) {
        acc = w_addp<F>(acc, w_load_pt<F>(part_tail + ts));
      } else if (__ldg(head_key + ts) != k) {
        if ((threadIdx.x & 31u) == 0) atomicOr(err, 1u);
      } else {
        acc = w_addp<F>(acc, w_load_pt<F>(part_head + ts));
      }
    }
    acc = w_block_sum<F>(acc, SUM_WARPS, w_smem + w_smem_bytes<F>(SUM_WARPS) / 4);
    if (w == 0) w_store_pt<F>(buckets + k, acc);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Window combination on the device, one block per MSM: result = sum_w
// 2^(c w) S_w by Horner; homogeneous projective output (u64 limbs,
// Montgomery).  The c (W - 1) doublings of the top window are one serial
// chain, run by Chain<F>::WARPS warps together (xyzz_chain.cuh).  The additions
// are kept off it: each of COMBINE_WARPS other warps combines a group of q
// windows, while the chain already works on the top 1 to q windows, and the
// chain takes in one sum every c q doublings (B200, against groups first and
// the chain after them: G1 1024 points 0.42 -> 0.39 ms, G2 1500 points
// 0.82 -> 0.65 ms, the chain's Fp2 products on 8 warps included).
// out_index (optional) maps MSM i to its result slot.  affine: an affine point
// of the reference's layout instead (infinity flag in the word after the
// coordinates).
// ---------------------------------------------------------------------------
template <class F>
__global__ void __launch_bounds__(COMBINE_THREADS<F>) k_combine(const xyzz_t<F> *__restrict__ S, int W, int c,
                                                                const int32_t *__restrict__ out_index,
                                                                uint64_t *__restrict__ out, bool affine) {
  using WP = WF<F>;
  constexpr int PT = w_pt_words<F>(), LW = WP::LW;
  w_setup();
  grid_wait(S);
  grid_release();
  const int64_t i = blockIdx.x;
  const int w = w_warp();
  constexpr int NCH = Chain<F>::WARPS, LEAD = COMBINE_WARPS;  // the chain's warps are LEAD .. LEAD + NCH - 1
  // top: the highest window with anything in it (scalars rarely reach the last ones)
  int top = 0;
  for (int b = 0; b < W; b += 32) {
    const int j = b + (int)(threadIdx.x & 31u);
    const unsigned m = __ballot_sync(0xffffffffu, j < W && !F::is_zero_raw(S[i * W + j].ZZ));
    if (m) top = b + 31 - __clz(m);
  }
  const int q = max(1, (top + COMBINE_WARPS - 1) / COMBINE_WARPS);
  const int groups = top / q;  // the windows from groups * q to top are the chain's own
  int32_t *sums = w_smem + w_smem_bytes<F>(LEAD + 1) / 4;
  int32_t *io = sums + COMBINE_WARPS * PT, *ctl = io + 3 * LW, *work = ctl + 4;
  wpt<F> res = w_inf<F>();
  if (w <= LEAD) {
    const int lo = w < LEAD ? w * q : groups * q, hi = w < LEAD ? (w + 1) * q : top + 1;
    if (w == LEAD || w < groups)
      for (int j = hi - 1; j >= lo; j--) {
        if (!res.inf)
          for (int k = 0; k < c; k++) res = w_dbl<F>(res);
        res = w_addp<F>(res, w_load_pt<F>(S + i * W + j));
      }
  }
  if (w < LEAD) {
    w_put_pt<F>(sums + w * PT, res);
    asm volatile("bar.arrive 2, %0;" ::"n"(COMBINE_THREADS<F>) : "memory");
    return;
  }
  bool waited = false;
  auto group_sums = [&] {  // once: the groups' warps are done
    if (!waited) asm volatile("bar.sync 2, %0;" ::"n"(COMBINE_THREADS<F>) : "memory");
    waited = true;
  };
  for (int j = groups - 1; j >= 0; j--) {
    if (w == LEAD) {
      if (threadIdx.x == 32 * LEAD) ctl[0] = res.inf ? 1 : 0;
      WP::put(io, res.X);
      WP::put(io + LW, res.Y);
      WP::put(io + 2 * LW, WP::one());
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NCH) : "memory");
    if (ctl[0] == 0) chain_dbl<F>(c * q, LEAD, io, work);
    group_sums();
    if (w == LEAD) {
      if (!res.inf) {
        const typename WP::E L = WP::get(io + 2 * LW);
        res.X = WP::get(io);
        res.Y = WP::get(io + LW);
        const int g = w_group();
        const typename WP::E t = WP::mul(WP::pick(g, L, res.ZZZ, L, L), L);
        const typename WP::E LL = WP::from(t, 0);
        const typename WP::E z = WP::mul(WP::pick(g, res.ZZ, WP::from(t, 1), LL, LL), LL);
        res.ZZ = WP::from(z, 0);
        res.ZZZ = WP::from(z, 1);
        if (WP::is_zero(L)) res = w_inf<F>();  // a point of order two was doubled
      }
      res = w_addp<F>(res, w_get_pt<F>(sums + j * PT));
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NCH) : "memory");
  }
  group_sums();  // where there are no groups the barrier is still to be completed
  if (w > LEAD) return;
  constexpr int H = F::LIMBS / 2;
  const int g = w_group();
  const int64_t slot = out_index ? (int64_t)__ldg(out_index + i) : i;
  if (res.inf) res = w_inf<F>();
  if (affine) {
    // x = X ZZZ I, y = Y ZZ I with I = 1 / (ZZ ZZZ); 0 for infinity
    const typename WP::E I = WP::inv(WP::mul(res.ZZ, res.ZZZ));
    const typename WP::E t = WP::mul(WP::pick(g, res.ZZZ, res.ZZ, res.ZZZ, res.ZZ), I);
    typename F::T v = WP::canon(WP::mul(WP::pick(g, res.X, res.Y, res.X, res.Y), t));
    uint64_t *o = out + slot * (2 * H + 1);
    if (g < 2 && w_lane() == 0) store_ref<F>(o + g * H, v);
    if (threadIdx.x == 32 * LEAD) o[2 * H] = res.inf ? 1u : 0u;
    return;
  }
  // (X ZZZ, Y ZZ, ZZ ZZZ); infinity is (0, 0, 0)
  const typename F::T o =
      WP::canon(WP::mul(WP::pick(g, res.X, res.Y, res.ZZ, res.ZZ), WP::pick(g, res.ZZZ, res.ZZ, res.ZZZ, res.ZZZ)));
  if (g < 3 && w_lane() == 0) {
    typename F::T v = o;
    store_ref<F>(out + (slot * 3 + g) * H, v);
  }
}

template <class F>
constexpr int combine_smem() {
  return w_smem_bytes<F>(COMBINE_WARPS + 1) + 4 * (COMBINE_WARPS * w_pt_words<F>() + 3 * WF<F>::LW + 4 + chain_words<F>());
}

// ---------------------------------------------------------------------------
// Host side: workspace layout and launch sequence of the reduction.
// ---------------------------------------------------------------------------
struct RedLayout {
  int64_t G = 0;
  int sms = 1, dev = 0;  // device the level-0 grid is sized for
  int B = 0, L0 = 0, nseg0 = 0, L1 = 0, nseg1 = 0, M = 0;
  bool warp0 = false;    // level 0 on warps
  size_t o_X = 0, o_A0 = 0, o_t[2] = {0, 0};

  // values per output of a sum stage over N values per group: up to 64 in one
  // block (8 additions per warp and the tree), else two stages of about sqrt(N)
  static int sum_chunk(int N) {
    if (N <= 64) return N;
    int q = 1;
    while (q * q < N) q++;
    return q;
  }

  // wave_threads: level-0 threads resident at once on the device.
  template <class F, class Carver>
  void plan(int64_t G_, int B_, int64_t wave_threads, int sms_, Carver &cv) {
    G = G_;
    B = B_;
    sms = sms_;
    // Level 0: on warps, about W_FILL warps per SM (they then fill its
    // schedulers), at least 4 buckets each; on threads when a resident wave of
    // threads would get more than RED_THREAD_MIN buckets each.
    const int64_t total = G * B;
    warp0 = wave_threads <= 0 || total <= RED_THREAD_MIN * wave_threads;
    int64_t l0;
    if (warp0)
      l0 = std::max<int64_t>(4, (total + (int64_t)sms * W_FILL - 1) / ((int64_t)sms * W_FILL));
    else
      l0 = (total + wave_threads - 1) / wave_threads;
    L0 = (int)std::min<int64_t>(l0, B);
    nseg0 = (B + L0 - 1) / L0;
    const int64_t l1 = std::max<int64_t>(4, (G * nseg0 + (int64_t)sms * W_FILL - 1) / ((int64_t)sms * W_FILL));
    L1 = (int)std::min<int64_t>(l1, nseg0);
    nseg1 = nseg0 > 1 ? (nseg0 + L1 - 1) / L1 : 0;
    M = nseg0 + nseg1;
    o_X = cv.template take<xyzz_t<F>>((size_t)(G * M));
    o_A0 = cv.template take<xyzz_t<F>>((size_t)(G * nseg0));
    int N = M;
    for (int k = 0; k < 2; k++) {
      const int ch = sum_chunk(N);
      N = (N + ch - 1) / ch;
      o_t[k] = cv.template take<xyzz_t<F>>((size_t)(G * N));
    }
  }
};

}  // namespace gm
