// MSM launch sequence (templated on the field), instantiated once per group
// in msm_g1.cu / msm_g2.cu so the two large kernel sets compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <cstring>
#include <string>
#include <vector>

#include "msm_engine.h"
#include "msm_affine.cuh"
#include "msm_kernels.cuh"
#include "msm_reduce.cuh"
#include "msm_sort.cuh"

namespace gm {

static inline int windows_for(int c, int limbs) { return (64 * limbs) / c + 1; }
#define GM_CHECK(call)                                     \
  do {                                                     \
    cudaError_t _e = (call);                               \
    if (_e != cudaSuccess) return record_error(_e, #call); \
  } while (0)

#define GM_CHECK_LAUNCH(where)                             \
  do {                                                     \
    cudaError_t _e = cudaGetLastError();                   \
    if (_e != cudaSuccess) return record_error(_e, where); \
  } while (0)

// ---------------------------------------------------------------------------
// workspace layout
// ---------------------------------------------------------------------------
static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct Carve {
  size_t off = 0;
  template <class T>
  size_t take(size_t count) {
    const size_t o = align_up(off, 256);
    off = o + count * sizeof(T);
    return o;
  }
};

// How the entries of an MSM (or of a batch class) are cut for accumulation.
// Warps: slices of ACC_WARP_MIN entries, of more once that would give more
// than W_FILL warps per SM, up to ACC_WARP_MAX entries on 4 times as many.
// Threads beyond: one slice per thread of a wave, of at least ACC_THREAD_MIN
// entries (shorter ones leave every bucket to the fix-up).  B200, one slice
// per thread at all sizes -> this rule, accumulation + fix-up: G1 1024 points
// 0.24 -> 0.12 ms, G2 1500 points 0.98 -> 0.37 ms, G1 4500 points 0.62 -> 0.30 ms.
// most: a caller's own bound on the slices (their partials' memory), or 0.
struct AccSlices {
  int64_t n = 0;
  bool warp = false;
};
static inline AccSlices acc_slices(int64_t max_entries, int64_t wave_threads, int sms, int64_t most = 0) {
  AccSlices a;
  const int64_t warps = (int64_t)sms * W_FILL;
  if (max_entries <= 4 * warps * ACC_WARP_MAX) {
    a.warp = true;
    const int64_t per = std::min<int64_t>(ACC_WARP_MAX, std::max<int64_t>(ACC_WARP_MIN, max_entries / warps));
    a.n = std::max<int64_t>(1, (max_entries + per - 1) / per);
  } else {
    a.n = std::min<int64_t>(std::max<int64_t>(128, wave_threads), (max_entries / ACC_THREAD_MIN + 127) / 128 * 128);
  }
  if (most > 0) a.n = std::min(a.n, most);
  return a;
}

template <class F>
struct MsmLayout {
  DigitParams dp;
  int64_t K = 0, nthreads = 0, n = 0;
  size_t o_offsets, o_entries, o_buckets, o_head, o_tail, o_hk, o_tk, o_err, o_packed, o_longq;
  size_t bytes = 0;
  int64_t long_cap = 0;
  bool need_pack = false;
  bool warp_acc = false;  // accumulation slices on warps
  AffLayout al;  // its scratch is not part of the workspace (ScratchLease)
  size_t o_aff = 0;
  SortLayout sl;
  RedLayout rl;

  // slice_threads: accumulation slices (one per thread of a single wave);
  // most_slices: bound on them, or 0;
  // level0_wave: threads of k_red_level0 resident at once
  void plan(int64_t n_, int limbs, int c, int64_t slice_threads, bool pack, int64_t level0_wave, int sms,
            int64_t most_slices, bool affine_rounds) {
    n = n_;
    need_pack = pack;
    dp.c = c;
    dp.W = windows_for(c, limbs);
    dp.B = 1 << (c - 1);
    dp.limbs = limbs;
    K = (int64_t)dp.W * dp.B;
    const int64_t max_entries = n * dp.W;
    const AccSlices as = acc_slices(max_entries, slice_threads, sms, most_slices);
    nthreads = as.n;
    warp_acc = as.warp;
    Carve cv;
    o_offsets = cv.take<uint32_t>(K + 1);
    o_entries = cv.take<uint32_t>((size_t)std::max<int64_t>(1, max_entries));
    sl.plan(dp, 1, n, (n + SA_TP - 1) / SA_TP, /*tabled=*/false, cv);
    o_buckets = cv.take<xyzz_t<F>>(K);
    o_head = cv.take<xyzz_t<F>>(nthreads);
    o_tail = cv.take<xyzz_t<F>>(nthreads);
    o_hk = cv.take<int32_t>(nthreads);
    o_tk = cv.take<int32_t>(nthreads);
    rl.plan<F>(dp.W, dp.B, level0_wave, sms, cv);
    long_cap = nthreads / FIX_SHORT + 1;
    o_longq = cv.take<int32_t>((size_t)(1 + long_cap));
    o_err = cv.take<uint32_t>(4);
    if (affine_rounds) al.plan<F, Carve>(&n, 1, dp.W, 1, dp.B, sms);
    o_aff = cv.take<char>(al.bytes);
    o_packed = pack ? cv.take<uint4>((size_t)n * Rec<F>::U4) : 0;
    bytes = cv.off;
  }
};

// k_accumulate runs at most ACC_BLOCKS_MAX blocks per SM.  Its slices carry
// equal work, so a block that shares its SM with more blocks than the others
// finishes late and holds up the whole launch: with 3 blocks per SM the G1
// 2^20 accumulation without affine rounds took 13.8 ms against 13.3 ms (with
// them 3 is slower again), and batches, whose classes'
// launches overlap, 196 ms against 143 ms.  The grid holds ACC_BLOCKS_MAX
// blocks per SM, and where the registers would let more blocks share an SM
// the launch asks for enough dynamic shared memory to keep them out.
constexpr int ACC_BLOCKS_MAX = 2;

struct AccOccupancy {
  int blocks = 0;     // resident blocks per SM the grid is sized for
  size_t smem = 0;    // dynamic shared memory of a launch
};

// which: 0 = k_accumulate<F>, 1 = k_accumulate_queue<F> (same limits)
template <class F>
static AccOccupancy acc_occupancy(int dev, int which = 0) {
  static std::mutex mu;
  static AccOccupancy cached[2][64];
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64) dev = 0;
  AccOccupancy &o = cached[which][dev];
  const void *fn = which == 0 ? (const void *)k_accumulate<F> : (const void *)k_accumulate_queue<F>;
  if (o.blocks == 0) {
    size_t smem = acc_smem_bytes<F>();
    int per_sm_smem = 0, b = 0;
    cudaDeviceGetAttribute(&per_sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, ACC_THREADS, smem) != cudaSuccess) b = 1;
    if (b > ACC_BLOCKS_MAX && per_sm_smem > 0) {
      // (ACC_BLOCKS_MAX + 1) blocks must not fit in the SM's shared memory
      const size_t pad = (size_t)per_sm_smem / (ACC_BLOCKS_MAX + 1) + 1024;
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pad) == cudaSuccess) smem = pad;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, ACC_THREADS, smem) != cudaSuccess) b = 1;
    }
    o.smem = smem;
    o.blocks = std::max(1, std::min(b, ACC_BLOCKS_MAX));
  }
  return o;
}

template <class F>
static int acc_blocks_per_sm(int dev) {
  return acc_occupancy<F>(dev).blocks;
}

template <class F>
static void acc_launch(bool warp, cudaStream_t s, const uint4 *bases, const uint32_t *entries,
                       const uint32_t *offsets, int64_t K, int64_t nthreads, xyzz_t<F> *buckets, xyzz_t<F> *head,
                       xyzz_t<F> *tail, int32_t *hk, int32_t *tk) {
  if (warp) {
    constexpr int WPB = W_THREADS / 32;
    launch_after(k_accumulate_warp<F>, (unsigned)((nthreads + WPB - 1) / WPB), W_THREADS, w_smem_bytes<F>(WPB), s,
                 bases, entries, offsets, K, nthreads, buckets, head, tail, hk, tk);
    return;
  }
  const unsigned grid = (unsigned)((nthreads + ACC_THREADS - 1) / ACC_THREADS);
  int dev = 0;
  cudaGetDevice(&dev);
  k_accumulate<F><<<grid, ACC_THREADS, acc_occupancy<F>(dev).smem, s>>>(bases, entries, offsets, K, nthreads,
                                                                          buckets, head, tail, hk, tk);
}

static inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

// Resident blocks per SM of the level-0 reduction kernel (cached per device).
template <class F>
static int level0_blocks_per_sm(int dev) {
  static std::mutex mu;
  static int cached[64] = {0};
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_red_level0<F>, 128, 0) != cudaSuccess) b = 1;
    cached[dev] = std::max(1, b);
  }
  return cached[dev];
}

// Split fix-up: short runs serially, long runs by a block-level tree.
// long_q[0] must be zero on entry.
template <class F>
int fixup_launch(cudaStream_t s, const uint32_t *offsets, int64_t K, int64_t nthreads, xyzz_t<F> *buckets,
                 const xyzz_t<F> *head, const xyzz_t<F> *tail, const int32_t *hk, const int32_t *tk, uint32_t *err,
                 int32_t *long_q, int64_t long_cap, int *launches) {
  launch_after(k_fixup_split<F>, grid_for(nthreads, W_THREADS / 32), W_THREADS, w_smem_bytes<F>(W_THREADS / 32), s,
               offsets, K, nthreads, buckets, head, tail, hk, tk, err, long_q, long_cap);
  GM_CHECK_LAUNCH("k_fixup_split");
  launch_after(k_fixup_long<F>, FIX_LONG_BLOCKS, 32 * SUM_WARPS, w_sum_smem<F>(SUM_WARPS), s, offsets, K, nthreads, buckets, head,
                                                                                    tail, hk, err, long_q, long_cap);
  GM_CHECK_LAUNCH("k_fixup_long");
  *launches += 2;
  return GM_OK;
}

// Leveled bucket reduction over rl.G groups of rl.B buckets; *sums receives
// the G window sums (contiguous).
template <class F>
int reduce_launch(cudaStream_t s, const RedLayout &rl, const xyzz_t<F> *buckets, const uint32_t *offsets, char *ws,
                  const xyzz_t<F> **sums, int *launches) {
  auto *X = (xyzz_t<F> *)(ws + rl.o_X);
  auto *A0 = (xyzz_t<F> *)(ws + rl.o_A0);
  constexpr int WPB = W_THREADS / 32;
  if (rl.warp0) {
    launch_after(k_red_level0_warp<F>, grid_for(rl.G * rl.nseg0, WPB), W_THREADS, w_smem_bytes<F>(WPB), s,
                 buckets, offsets, rl.G, rl.B, rl.L0, rl.nseg0, X, rl.M, A0);
  } else {
    const int64_t wave = (int64_t)rl.sms * level0_blocks_per_sm<F>(rl.dev);
    const int64_t blocks0 = std::min<int64_t>(wave, (rl.G * rl.nseg0 + 127) / 128);
    k_red_level0<F><<<(unsigned)std::max<int64_t>(1, blocks0), 128, 0, s>>>(buckets, offsets, rl.G, rl.B, rl.L0,
                                                                             rl.nseg0, X, rl.M, A0);
  }
  GM_CHECK_LAUNCH("k_red_level0");
  (*launches)++;
  if (rl.nseg1 > 0) {
    launch_after(k_red_level1<F>, grid_for(rl.G * rl.nseg1, WPB), W_THREADS, w_smem_bytes<F>(WPB), s,
                 A0, rl.G, rl.nseg0, rl.L1, rl.nseg1, rl.L0, X, rl.M);
    GM_CHECK_LAUNCH("k_red_level1");
    (*launches)++;
  }
  const xyzz_t<F> *src = X;
  int N = rl.M, k = 0;
  while (N > 1) {
    const int chunk = RedLayout::sum_chunk(N), nout = (N + chunk - 1) / chunk;
    auto *dst = (xyzz_t<F> *)(ws + rl.o_t[k]);
    launch_after(k_red_sum<F>, (unsigned)(rl.G * nout), 32 * SUM_WARPS, w_sum_smem<F>(SUM_WARPS), s, src, N, chunk, nout, dst);
    GM_CHECK_LAUNCH("k_red_sum");
    (*launches)++;
    src = dst;
    k ^= 1;
    N = nout;
  }
  *sums = src;
  return GM_OK;
}

// Plans the workspace of one MSM on device dev.  slice_threads 0: one
// accumulation slice per thread of a full wave (ACC_BLOCKS_MAX blocks per SM)
// or per warp (acc_slices); else at most that many slices.
template <class F>
int msm_plan(MsmLayout<F> &lay, int dev, int64_t n, int limbs, int c, bool pack, int64_t slice_threads,
             bool affine_rounds) {
  if (limbs < 1 || limbs > MAX_SCALAR_LIMBS || n < 1 || n > (int64_t)INT32_MAX) {
    set_last_error("invalid scalar_limbs or n");
    return GM_ERR_ARG;
  }
  if (c < 2 || c > 20) {
    set_last_error("window width out of range");
    return GM_ERR_ARG;
  }
  int sms = 0;
  int rc = device_sm_count(dev, &sms);
  if (rc) return rc;
  const int64_t most = slice_threads;
  if (slice_threads <= 0) slice_threads = (int64_t)sms * acc_blocks_per_sm<F>(dev) * ACC_THREADS;
  lay.plan(n, limbs, c, slice_threads, pack, (int64_t)sms * level0_blocks_per_sm<F>(dev) * 128, sms, most,
           affine_rounds);
  lay.rl.dev = dev;
  if ((uint64_t)n * lay.dp.W >= (1ull << 32)) {
    set_last_error("too many (point, window) entries for 32-bit offsets");
    return GM_ERR_ARG;
  }
  return GM_OK;
}

// Enqueues the whole pipeline of one planned MSM on s, in the workspace ws
// (lay.bytes, 256-byte aligned); allocates nothing itself, except that the
// affine rounds, where planned, run in a scratch block if the device has room for one.  bases: packed
// records, or null to pack from ref_points (reference layout; to_mont converts
// standard-form points).  out receives the result in the reference layout,
// projective or (affine) affine.  err_out (optional,
// device) receives the consistency flag of the fix-up (0 = ok).  bases_ready
// (optional): an event the stream waits for after the sort, before the bases
// are first read.  handoff (optional): the window sums are copied to the
// caller's pinned buffer instead, and out is not written.
template <class F>
int msm_run(cudaStream_t s, const MsmLayout<F> &lay, char *ws, const uint4 *bases, const uint64_t *ref_points,
            int to_mont, const uint64_t *scalars, uint64_t *out, uint32_t *err_out, cudaEvent_t bases_ready,
            TailHandoff *handoff = nullptr, bool affine = false) {
  constexpr int H = F::LIMBS / 2;  // u64 words per coordinate
  const int64_t n = lay.n;
  auto *sorted_off = (uint32_t *)(ws + lay.o_offsets);
  auto *sorted = (uint32_t *)(ws + lay.o_entries);
  const uint32_t *offsets = sorted_off, *entries = sorted;
  auto *buckets = (xyzz_t<F> *)(ws + lay.o_buckets);
  auto *head = (xyzz_t<F> *)(ws + lay.o_head);
  auto *tail = (xyzz_t<F> *)(ws + lay.o_tail);
  auto *hk = (int32_t *)(ws + lay.o_hk);
  auto *tk = (int32_t *)(ws + lay.o_tk);
  auto *err = (uint32_t *)(ws + lay.o_err);
  auto *long_q = (int32_t *)(ws + lay.o_longq);
  profile_mark(s, "start");
  int launches = 0;
  // the sort needs only the scalars; the bases are packed after it, so a
  // caller that is still copying them in can overlap that copy with the sort
  GM_CHECK(cudaMemsetAsync(err, 0, sizeof(uint32_t), s));
  GM_CHECK(cudaMemsetAsync(long_q, 0, sizeof(int32_t), s));
  {
    SortDesc sd;
    sd.n_single = n;
    const cudaError_t e = sort_launch(s, lay.sl, ws, scalars, sd, lay.K, sorted_off, sorted, &launches);
    if (e != cudaSuccess) return record_error(e, "sort");
  }
  profile_mark(s, "sort");
  if (bases_ready) GM_CHECK(cudaStreamWaitEvent(s, bases_ready, 0));
  if (bases == nullptr) {
    uint4 *packed = (uint4 *)(ws + lay.o_packed);
    k_pack_ref<F><<<grid_for(n, 256), 256, 0, s>>>(packed, ref_points, n, 2 * H + 1, to_mont);
    GM_CHECK_LAUNCH("k_pack_ref");
    bases = packed;
    launches++;
    profile_mark(s, "pack");
  }
  if (lay.al.rounds > 0) {
    ScratchLease lease;
    if (char *scratch = lease.acquire(lay.rl.dev, s, lay.al.scratch)) {
      const cudaError_t e = aff_launch<F>(s, lay.al, ws + lay.o_aff, scratch, bases, entries, offsets, &launches);
      if (e != cudaSuccess) return record_error(e, "k_affine_round");
      profile_mark(s, "affine");
      bases = lay.al.final_points(ws + lay.o_aff);
      entries = nullptr;
      offsets = lay.al.final_offsets(ws + lay.o_aff);
    }
  }
  acc_launch<F>(lay.warp_acc, s, bases, entries, offsets, lay.K, lay.nthreads, buckets, head, tail, hk, tk);
  GM_CHECK_LAUNCH("k_accumulate");
  launches++;
  profile_mark(s, "accumulate");
  int rc = fixup_launch<F>(s, offsets, lay.K, lay.nthreads, buckets, head, tail, hk, tk, err, long_q, lay.long_cap,
                           &launches);
  if (rc) return rc;
  profile_mark(s, "fixup");

  // bucket reduction: leveled running sums, then block sums
  const int W = lay.dp.W;
  const xyzz_t<F> *src = nullptr;
  rc = reduce_launch<F>(s, lay.rl, buckets, offsets, ws, &src, &launches);
  if (rc) return rc;
  profile_mark(s, "reduce");
  if (handoff) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GM_CHECK(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
      set_last_error("window-sum handoff while the stream is being captured");
      return GM_ERR_ARG;
    }
    const size_t bytes = (size_t)W * sizeof(xyzz_t<F>);
    if (bytes > handoff->cap) {
      set_last_error("window-sum handoff buffer too small");
      return GM_ERR_ARG;
    }
    GM_CHECK(cudaMemcpyAsync(handoff->host, src, bytes, cudaMemcpyDeviceToHost, s));
    handoff->W = W;
    handoff->c = lay.dp.c;
  } else {
    launch_after(k_combine<F>, 1, COMBINE_THREADS<F>, combine_smem<F>(), s, src, W, lay.dp.c, nullptr, out,
                                                                                    affine);
    GM_CHECK_LAUNCH("k_combine");
    launches++;
  }
  profile_mark(s, "combine");
  count_launches(launches);
  if (err_out) GM_CHECK(cudaMemcpyAsync(err_out, err, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  return GM_OK;
}

// The whole pipeline with its workspace from the device's stream-ordered
// pool, released on s after the last kernel (also when an enqueue fails).
// c_override 0: the window width from the cost model.
template <class F>
int msm_launch(cudaStream_t s, int dev, const uint4 *bases, const uint64_t *ref_points, int to_mont,
               const uint64_t *scalars, int limbs, int64_t n, uint64_t *out, int c_override,
               uint32_t *err_out, cudaEvent_t bases_ready, TailHandoff *handoff, bool affine) {
  constexpr int H = F::LIMBS / 2;
  if (n == 0) {
    if (err_out) GM_CHECK(cudaMemsetAsync(err_out, 0, sizeof(uint32_t), s));
    GM_CHECK(cudaMemsetAsync(out, 0, (affine ? 2 * H + 1 : 3 * H) * sizeof(uint64_t), s));
    if (affine) GM_CHECK(cudaMemsetAsync(out + 2 * H, 1, 1, s));  // infinity
    return GM_OK;
  }
  const int c = c_override > 0 ? c_override : default_window(sizeof(typename F::T) == sizeof(fp_t) ? 1 : 2, n, limbs);
  // without the affine rounds where the device has no room for what they leave
  MsmLayout<F> lay;
  char *ws = nullptr;
  int rc = GM_OK;
  for (const bool rounds : {true, false}) {
    lay = MsmLayout<F>();
    rc = msm_plan<F>(lay, dev, n, limbs, c, bases == nullptr, 0, rounds);
    if (rc) return rc;
    rc = pool_alloc(dev, s, lay.bytes, (void **)&ws);
    if (rc == GM_OK || lay.al.rounds == 0) break;
    cudaGetLastError();  // the failed allocation
  }
  if (rc) return rc;
  rc = msm_run<F>(s, lay, ws, bases, ref_points, to_mont, scalars, out, err_out, bases_ready,
                  handoff, affine);
  const cudaError_t e = cudaFreeAsync(ws, s);
  if (rc) return rc;
  return e == cudaSuccess ? GM_OK : record_error(e, "cudaFreeAsync(workspace)");
}

}  // namespace gm
