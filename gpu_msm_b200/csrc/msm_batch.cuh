// Batched MSM engine: many independent MSMs of uneven size over one resident
// base table, executed as one flattened pipeline per window-width class.
//
// A plan fixes the batch's shape (sizes, base offsets, window width per MSM),
// groups the MSMs into classes of equal window width, uploads the per-MSM
// descriptors and allocates every workspace once.  Running the plan only
// enqueues kernels and memsets: each class on its own stream, forked from and
// joined back to the caller's stream with events, so a run can be captured
// into a CUDA graph and replayed with new scalars in the same buffer.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "msm_host.cuh"

namespace gm {

struct BatchClassPlan {
  int c = 0;
  DigitParams dp{};
  int count = 0;        // MSMs in this class
  std::vector<int64_t> sizes;  // their points
  int64_t P = 0;        // points in this class
  int64_t K = 0, nthreads = 0;
  bool warp_acc = false;  // accumulation slices on warps (then outside the queued launch)
  int64_t tilesA = 0;   // pass-A sort tiles (SA_THREADS * sort_ppt points, one MSM each)
  int slice_waves = 1;  // accumulation slices: this many resident waves of threads
  int sort_ppt = SA_PPT;  // pass-A sort tile: points per thread (2, 4 or 8)
  SortLayout sl;
  RedLayout rl;
  int64_t long_cap = 0;
  // fixed-base window table (precomputed mode): record w*pc_stride + base
  const uint4 *pc_table = nullptr;
  int64_t pc_stride = 0;
  size_t o_offsets = 0, o_entries = 0, o_buckets = 0, o_head = 0, o_tail = 0, o_hk = 0, o_tk = 0, o_longq = 0,
         o_err = 0;
  size_t ws_bytes = 0;
  char *ws = nullptr;       // workspace (owned)
  // rounds of affine additions; used where aff_ws and the plan's aff_scratch are there
  AffLayout al;
  char *aff_ws = nullptr;   // al.bytes (owned)
  // descriptors (owned): int64 point_start[count+1] | base_off[count] |
  // sc_off[count], then int32 out_index[count] | tile_first[count+1]
  char *desc = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;
  cudaEvent_t sorted = nullptr;  // queued accumulation: this class's sort has run
};

struct BatchPlan {
  int group = 1, dev = 0, limbs = 1, count = 0;
  const uint4 *bases = nullptr;
  int64_t n_bases = 0;
  std::vector<BatchClassPlan> classes;
  cudaEvent_t fork = nullptr;
  size_t bytes = 0;
  // scratch of the affine rounds, which run class after class: owned, or (lease) a scratch block for each class
  char *aff_scratch = nullptr;
  bool lease = false;
  size_t aff_scratch_bytes() const {
    size_t b = 0;
    for (const auto &cp : classes) b = std::max(b, cp.al.scratch);
    return b;
  }
  bool rounds(const BatchClassPlan &cp) const { return cp.al.rounds > 0 && cp.aff_ws && (aff_scratch || lease); }
  // Accumulation mode of plans: true (default) = every class's accumulation
  // in one persistent launch over a device work queue (k_accumulate_queue)
  // between the classes' sorts and their fix-ups; false = one pipeline per
  // class on its own stream, every kernel of a class a full-GPU launch.
  // The 512-MSM batch (2^8..2^16 points, 2^16-point table) measured 97.7 ms
  // queued against 99.2 ms per class on B200, and 67.0 against 67.5 ms with
  // fixed-base window tables.  Transient batches
  // (gm_batch_run) run their classes in order on the caller's stream.
  bool queue = true;
  char *acc_desc = nullptr;      // AccClass<F>[classes] (owned)
  uint32_t *queue_ctr = nullptr; // work-queue counter (owned)
  int64_t queue_items = 0;
  cudaEvent_t acc_done = nullptr;
};

// Workspace layout of one class (same parts as a single MSM, K over all the
// class's MSMs, no base packing).
template <class F>
void batch_class_layout(BatchClassPlan &cp, int limbs, int sms, int dev) {
  cp.dp.c = cp.c;
  cp.dp.W = windows_for(cp.c, limbs);
  cp.dp.B = 1 << (cp.c - 1);
  cp.dp.limbs = limbs;
  // precomputed mode: one bucket set per MSM (no window index in the key)
  const int64_t groups = (int64_t)cp.count * (cp.pc_stride ? 1 : cp.dp.W);
  cp.K = groups * cp.dp.B;
  const int64_t max_entries = cp.P * cp.dp.W;
  const AccSlices as =
      acc_slices(max_entries, (int64_t)sms * acc_blocks_per_sm<F>(dev) * ACC_THREADS * cp.slice_waves, sms);
  cp.nthreads = as.n;
  cp.warp_acc = as.warp;
  Carve cv;
  cp.o_offsets = cv.take<uint32_t>(cp.K + 1);
  cp.o_entries = cv.take<uint32_t>((size_t)std::max<int64_t>(1, max_entries));
  cp.sl.plan(cp.dp, cp.count, cp.P, cp.tilesA, cp.pc_stride != 0, cv, cp.sort_ppt);
  cp.o_buckets = cv.take<xyzz_t<F>>(cp.K);
  cp.o_head = cv.take<xyzz_t<F>>(cp.nthreads);
  cp.o_tail = cv.take<xyzz_t<F>>(cp.nthreads);
  cp.o_hk = cv.take<int32_t>(cp.nthreads);
  cp.o_tk = cv.take<int32_t>(cp.nthreads);
  cp.rl.plan<F>(groups, cp.dp.B, (int64_t)sms * level0_blocks_per_sm<F>(dev) * 128, sms, cv);
  cp.rl.dev = dev;
  cp.long_cap = cp.nthreads / FIX_SHORT + 1;
  cp.o_longq = cv.take<int32_t>((size_t)(1 + cp.long_cap));
  cp.o_err = cv.take<uint32_t>(4);
  cp.ws_bytes = cv.off;
  cp.al = AffLayout();
  if (!cp.warp_acc)
    cp.al.plan<F, Carve>(cp.sizes.data(), cp.count, cp.pc_stride ? 1 : cp.dp.W, cp.pc_stride ? cp.dp.W : 1, cp.dp.B,
                         sms);
}

// Pointers into one class's workspace.
template <class F>
struct ClassBufs {
  uint32_t *offsets, *entries, *err;
  // what is accumulated: the sorted entries over the bases, or what the affine rounds leave
  const uint4 *acc_bases;
  const uint32_t *acc_entries, *acc_offsets;
  int32_t *hk, *tk, *long_q;
  xyzz_t<F> *buckets, *head, *tail;
  SortDesc sd;
  const int32_t *out_index;
  ClassBufs(const BatchPlan &plan, const BatchClassPlan &cp, bool rounds) {
    char *ws = cp.ws;
    offsets = (uint32_t *)(ws + cp.o_offsets);
    entries = (uint32_t *)(ws + cp.o_entries);
    buckets = (xyzz_t<F> *)(ws + cp.o_buckets);
    head = (xyzz_t<F> *)(ws + cp.o_head);
    tail = (xyzz_t<F> *)(ws + cp.o_tail);
    hk = (int32_t *)(ws + cp.o_hk);
    tk = (int32_t *)(ws + cp.o_tk);
    err = (uint32_t *)(ws + cp.o_err);
    long_q = (int32_t *)(ws + cp.o_longq);
    acc_bases = cp.pc_table ? cp.pc_table : plan.bases;
    acc_entries = entries;
    acc_offsets = offsets;
    if (rounds) {
      acc_bases = cp.al.final_points(cp.aff_ws);
      acc_entries = nullptr;
      acc_offsets = cp.al.final_offsets(cp.aff_ws);
    }
    sd.point_start = (const int64_t *)cp.desc;
    sd.base_off = sd.point_start + cp.count + 1;
    sd.sc_off = sd.base_off + cp.count;
    sd.count = cp.count;
    sd.pc_stride = cp.pc_stride;
    out_index = (const int32_t *)(sd.sc_off + cp.count);
    sd.tile_first = out_index + cp.count;
  }
};

// One class, first part: flags cleared, entries sorted.
template <class F>
int batch_class_sort(const BatchPlan &plan, const BatchClassPlan &cp, cudaStream_t s, const uint64_t *scalars,
                     int *launches) {
  ClassBufs<F> cb(plan, cp, false);
  GM_CHECK(cudaMemsetAsync(cb.err, 0, sizeof(uint32_t), s));
  GM_CHECK(cudaMemsetAsync(cb.long_q, 0, sizeof(int32_t), s));
  const cudaError_t e = sort_launch(s, cp.sl, cp.ws, scalars, cb.sd, cp.K, cb.offsets, cb.entries, launches);
  if (e != cudaSuccess) return record_error(e, "batch sort");
  return GM_OK;
}

// One class, last part (after its accumulation): fix-up, reduction, and the
// window combination into the class's result slots.
template <class F>
int batch_class_finish(const BatchPlan &plan, const BatchClassPlan &cp, cudaStream_t s, bool rounds, uint64_t *results,
                       int *launches) {
  ClassBufs<F> cb(plan, cp, rounds);
  int rc = fixup_launch<F>(s, cb.acc_offsets, cp.K, cp.nthreads, cb.buckets, cb.head, cb.tail, cb.hk, cb.tk, cb.err,
                           cb.long_q, cp.long_cap, launches);
  if (rc) return rc;
  const xyzz_t<F> *src = nullptr;
  rc = reduce_launch<F>(s, cp.rl, cb.buckets, cb.acc_offsets, cp.ws, &src, launches);
  if (rc) return rc;
  // precomputed mode: one window per MSM, so the combination is a conversion
  launch_after(
      k_combine<F>, (unsigned)cp.count, COMBINE_THREADS<F>, combine_smem<F>(), s, src, cp.pc_stride ? 1 : cp.dp.W, cp.c, cb.out_index, results, false);
  GM_CHECK_LAUNCH("k_combine");
  (*launches)++;
  return GM_OK;
}

// One class, the affine rounds over its sorted entries.  *ran: false where no
// scratch block could be had (never with the plan's own scratch).
template <class F>
int batch_class_rounds(const BatchPlan &plan, const BatchClassPlan &cp, cudaStream_t s, int *launches, bool *ran) {
  ClassBufs<F> cb(plan, cp, false);
  ScratchLease lease;
  char *scratch = plan.aff_scratch ? plan.aff_scratch : lease.acquire(plan.dev, s, cp.al.scratch);
  *ran = scratch != nullptr;
  if (!scratch) return GM_OK;
  const cudaError_t e = aff_launch<F>(s, cp.al, cp.aff_ws, scratch, cb.acc_bases, cb.acc_entries, cb.acc_offsets,
                                      launches);
  return e == cudaSuccess ? GM_OK : record_error(e, "k_affine_round");
}

template <class F>
int batch_class_accumulate(const BatchPlan &plan, const BatchClassPlan &cp, cudaStream_t s, bool rounds,
                           int *launches) {
  ClassBufs<F> cb(plan, cp, rounds);
  acc_launch<F>(cp.warp_acc, s, cb.acc_bases, cb.acc_entries, cb.acc_offsets, cp.K, cp.nthreads, cb.buckets, cb.head,
                cb.tail, cb.hk, cb.tk);
  GM_CHECK_LAUNCH("k_accumulate");
  (*launches)++;
  return GM_OK;
}

// Enqueue one class's whole pipeline on `s`.
template <class F>
int batch_class_run(const BatchPlan &plan, const BatchClassPlan &cp, cudaStream_t s, const uint64_t *scalars,
                    uint64_t *results) {
  if (cp.count == 0) return GM_OK;
  int launches = 0;
  int rc = batch_class_sort<F>(plan, cp, s, scalars, &launches);
  if (rc) return rc;
  bool rounds = plan.rounds(cp);
  if (rounds) rc = batch_class_rounds<F>(plan, cp, s, &launches, &rounds);
  if (rc) return rc;
  rc = batch_class_accumulate<F>(plan, cp, s, rounds, &launches);
  if (rc) return rc;
  rc = batch_class_finish<F>(plan, cp, s, rounds, results, &launches);
  count_launches(launches);
  return rc;
}

// Device descriptors of the queued accumulation (plans with their own
// streams): one AccClass per class, written into plan.acc_desc.
template <class F>
int batch_queue_setup(BatchPlan &plan) {
  std::vector<AccClass<F>> h(plan.classes.size());
  int64_t items = 0;
  for (size_t k = 0; k < plan.classes.size(); k++) {
    const BatchClassPlan &cp = plan.classes[k];
    ClassBufs<F> cb(plan, cp, plan.rounds(cp));
    h[k] = AccClass<F>{cb.acc_bases, cb.acc_entries, cb.acc_offsets, cp.K, cp.nthreads,
                       cb.buckets, cb.head, cb.tail, cb.hk, cb.tk, items};
    if (!cp.warp_acc) items += cp.nthreads / 32;  // nthreads is a multiple of 128 then
  }
  plan.queue_items = items;
  GM_CHECK(cudaMemcpy(plan.acc_desc, h.data(), h.size() * sizeof(AccClass<F>), cudaMemcpyHostToDevice));
  return GM_OK;
}

// The queued flow: every class sorts on its stream; s joins them, runs the
// affine rounds class after class and the accumulation of all classes in one
// persistent launch, and forks the
// classes again for their fix-ups, reductions and combinations.
template <class F>
int batch_run_queued(const BatchPlan &plan, cudaStream_t s, const uint64_t *scalars, uint64_t *results) {
  int launches = 0;
  GM_CHECK(cudaEventRecord(plan.fork, s));
  for (const auto &cp : plan.classes) {
    GM_CHECK(cudaStreamWaitEvent(cp.stream, plan.fork, 0));
    int rc = batch_class_sort<F>(plan, cp, cp.stream, scalars, &launches);
    if (rc) return rc;
    if (cp.warp_acc) {  // few entries: the class's whole pipeline beside the others
      rc = batch_class_accumulate<F>(plan, cp, cp.stream, false, &launches);
      if (rc) return rc;
      rc = batch_class_finish<F>(plan, cp, cp.stream, false, results, &launches);
      if (rc) return rc;
    }
    GM_CHECK(cudaEventRecord(cp.sorted, cp.stream));
    GM_CHECK(cudaStreamWaitEvent(s, cp.sorted, 0));
  }
  if (plan.queue_items == 0) {
    count_launches(launches);
    return GM_OK;
  }
  int rc = GM_OK;
  bool ran = false;
  for (const auto &cp : plan.classes)
    if (plan.rounds(cp)) {
      rc = batch_class_rounds<F>(plan, cp, s, &launches, &ran);
      if (rc) return rc;
    }
  GM_CHECK(cudaMemsetAsync(plan.queue_ctr, 0, sizeof(uint32_t), s));
  int dev = 0, sms = 0;
  GM_CHECK(cudaGetDevice(&dev));
  rc = device_sm_count(dev, &sms);
  if (rc) return rc;
  const AccOccupancy occ = acc_occupancy<F>(dev, 1);
  k_accumulate_queue<F><<<(unsigned)(sms * occ.blocks), ACC_THREADS, occ.smem, s>>>(
      (const AccClass<F> *)plan.acc_desc, (int)plan.classes.size(), plan.queue_items, plan.queue_ctr);
  GM_CHECK_LAUNCH("k_accumulate_queue");
  launches++;
  GM_CHECK(cudaEventRecord(plan.acc_done, s));
  for (const auto &cp : plan.classes) {
    if (cp.warp_acc) continue;
    GM_CHECK(cudaStreamWaitEvent(cp.stream, plan.acc_done, 0));
    rc = batch_class_finish<F>(plan, cp, cp.stream, plan.rounds(cp), results, &launches);
    if (rc) return rc;
    GM_CHECK(cudaEventRecord(cp.done, cp.stream));
    GM_CHECK(cudaStreamWaitEvent(s, cp.done, 0));
  }
  count_launches(launches);
  return GM_OK;
}

// Builds the fixed-base window table of n packed points: W windows of c bits.
template <class F>
int window_table_launch(cudaStream_t s, const uint4 *packed, int64_t n, int c, int W, uint4 *table) {
  k_window_table<F><<<grid_for(n, 128), 128, 0, s>>>(packed, n, c, W, table);
  GM_CHECK_LAUNCH("k_window_table");
  count_launches(1);
  return GM_OK;
}

template <class F>
int batch_layouts(BatchPlan &plan, int sms) {
  for (auto &cp : plan.classes) batch_class_layout<F>(cp, plan.limbs, sms, plan.dev);
  return GM_OK;
}

// Every class's pipeline on its own stream, forked from and joined back to s.
// The classes share the affine rounds' scratch, so those run on s, class after
// class; the rest of a class with rounds follows them on its stream.  Slices and
// rounds are those of the queued flow: the results agree word for word.
template <class F>
int batch_run_classes(const BatchPlan &plan, cudaStream_t s, const uint64_t *scalars, uint64_t *results) {
  int launches = 0, rc = GM_OK;
  bool ran = false;
  GM_CHECK(cudaEventRecord(plan.fork, s));
  for (const auto &cp : plan.classes) {
    GM_CHECK(cudaStreamWaitEvent(cp.stream, plan.fork, 0));
    rc = batch_class_sort<F>(plan, cp, cp.stream, scalars, &launches);
    if (rc) return rc;
    if (plan.rounds(cp)) {
      GM_CHECK(cudaEventRecord(cp.sorted, cp.stream));
      continue;
    }
    rc = batch_class_accumulate<F>(plan, cp, cp.stream, false, &launches);
    if (rc) return rc;
    rc = batch_class_finish<F>(plan, cp, cp.stream, false, results, &launches);
    if (rc) return rc;
  }
  for (const auto &cp : plan.classes) {
    if (!plan.rounds(cp)) continue;
    GM_CHECK(cudaStreamWaitEvent(s, cp.sorted, 0));
    rc = batch_class_rounds<F>(plan, cp, s, &launches, &ran);
    if (rc) return rc;
    GM_CHECK(cudaEventRecord(cp.done, s));
    GM_CHECK(cudaStreamWaitEvent(cp.stream, cp.done, 0));
    rc = batch_class_accumulate<F>(plan, cp, cp.stream, true, &launches);
    if (rc) return rc;
    rc = batch_class_finish<F>(plan, cp, cp.stream, true, results, &launches);
    if (rc) return rc;
  }
  for (const auto &cp : plan.classes) {
    GM_CHECK(cudaEventRecord(cp.done, cp.stream));
    GM_CHECK(cudaStreamWaitEvent(s, cp.done, 0));
  }
  count_launches(launches);
  return GM_OK;
}

// Fork the classes onto their streams and join them back into `s` (plans
// with their own streams), or run them in order on `s`.
template <class F>
int batch_run(const BatchPlan &plan, cudaStream_t s, const uint64_t *scalars, uint64_t *results) {
  if (plan.classes.size() == 1 || plan.fork == nullptr) {
    // one class, or a transient plan without its own streams: in order on s
    for (const auto &cp : plan.classes) {
      const int rc = batch_class_run<F>(plan, cp, s, scalars, results);
      if (rc) return rc;
    }
    return GM_OK;
  }
  if (plan.queue && plan.acc_desc) return batch_run_queued<F>(plan, s, scalars, results);
  return batch_run_classes<F>(plan, s, scalars, results);
}

}  // namespace gm
