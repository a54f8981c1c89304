// Host side of the MSM engine shared by both groups: error bookkeeping,
// per-device state and memory pool, window selection.
//
// Replaces the reference's MSM drivers (pdroalves/gpu_msm src/curve.cu:2538-2826)
// and C wrappers (rust-api/src/c_wrapper.cu).  Unlike the reference, which
// copies 16 buckets to the host and blocks three times per window, the whole
// MSM here is one asynchronous launch sequence on the caller's stream with no
// host round trip; workspace comes from a per-device stream-ordered memory
// pool so concurrent calls on different streams never share scratch.
#include <cuda_runtime.h>

#include <cstdlib>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/gpu_msm_b200.h"
#include "msm_engine.h"

namespace gm {

// ---------------------------------------------------------------------------
// error bookkeeping
// ---------------------------------------------------------------------------
static thread_local std::string g_last_error = "";

int record_error(cudaError_t e, const char *where) {
  g_last_error = std::string(where) + ": " + cudaGetErrorString(e);
  return GM_ERR_CUDA;
}

const char *last_error() { return g_last_error.c_str(); }

void set_last_error(const char *msg) { g_last_error = msg; }

#define GM_CHECK(call)                                                  \
  do {                                                                  \
    cudaError_t _e = (call);                                            \
    if (_e != cudaSuccess) return record_error(_e, #call);              \
  } while (0)

#define GM_CHECK_LAUNCH(where)                                          \
  do {                                                                  \
    cudaError_t _e = cudaGetLastError();                                \
    if (_e != cudaSuccess) return record_error(_e, where);              \
  } while (0)

// ---------------------------------------------------------------------------
// per-device state: SM count and a stream-ordered pool that keeps memory
// cached between calls (release threshold = unlimited)
// ---------------------------------------------------------------------------
struct DeviceState {
  int sms = 0;
  cudaMemPool_t pool = nullptr;
};

static std::mutex g_dev_mu;
static std::map<int, DeviceState> g_dev;

int device_state(int dev, DeviceState **out) {
  std::lock_guard<std::mutex> lk(g_dev_mu);
  auto it = g_dev.find(dev);
  if (it == g_dev.end()) {
    DeviceState st;
    GM_CHECK(cudaDeviceGetAttribute(&st.sms, cudaDevAttrMultiProcessorCount, dev));
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    GM_CHECK(cudaMemPoolCreate(&st.pool, &props));
    uint64_t thr = UINT64_MAX;
    GM_CHECK(cudaMemPoolSetAttribute(st.pool, cudaMemPoolAttrReleaseThreshold, &thr));
    it = g_dev.emplace(dev, st).first;
  }
  *out = &it->second;
  return GM_OK;
}

// ---------------------------------------------------------------------------
// phase profiling (CUDA events on the launching stream) and launch counting,
// per host thread
// ---------------------------------------------------------------------------
struct PhaseMark {
  const char *name;
  cudaEvent_t ev;
};
static thread_local bool g_prof_on = false;
static thread_local std::vector<PhaseMark> g_marks;
static thread_local std::vector<std::pair<std::string, float>> g_phase_ms;
static thread_local int64_t g_launches = 0;

void profile_enable(bool on) { g_prof_on = on; }
bool profile_enabled() { return g_prof_on; }

void profile_mark(cudaStream_t s, const char *name) {
  if (!g_prof_on) return;
  PhaseMark m{name, nullptr};
  if (cudaEventCreate(&m.ev) != cudaSuccess) return;
  cudaEventRecord(m.ev, s);
  g_marks.push_back(m);
}

// Closes the marks of one call: consecutive marks delimit phases.
void profile_end_call() {
  if (!g_prof_on) return;
  for (size_t i = 1; i < g_marks.size(); i++) {
    float ms = 0.f;
    cudaEventSynchronize(g_marks[i].ev);
    cudaEventElapsedTime(&ms, g_marks[i - 1].ev, g_marks[i].ev);
    g_phase_ms.emplace_back(g_marks[i].name, ms);
  }
  for (auto &m : g_marks) cudaEventDestroy(m.ev);
  g_marks.clear();
}

int profile_collect(char *names, int names_len, float *ms, int max) {
  profile_end_call();
  int n = 0;
  std::string joined;
  for (auto &p : g_phase_ms) {
    if (n < max) {
      ms[n] = p.second;
      if (!joined.empty()) joined += ",";
      joined += p.first;
    }
    n++;
  }
  if (names && names_len > 0) {
    strncpy(names, joined.c_str(), names_len - 1);
    names[names_len - 1] = 0;
  }
  g_phase_ms.clear();
  return n < max ? n : max;
}

void count_launches(int k) { g_launches += k; }
int64_t launches_and_reset() {
  const int64_t v = g_launches;
  g_launches = 0;
  return v;
}

// ---------------------------------------------------------------------------
// pinned host slots (descriptors, window sums and results on their way)
// ---------------------------------------------------------------------------
static std::mutex g_pin_mu;
static std::vector<void *> g_pin_free;
// Slots whose last copy is still pending: returned to the free list once
// their event has completed.  A host function per release would cost a
// driver round trip (~0.2 ms of stream time) for nothing.
struct PendingSlot {
  void *slot;
  cudaEvent_t ev;
  int dev;
};
static std::vector<PendingSlot> g_pin_pending;
static std::map<int, std::vector<cudaEvent_t>> g_free_events;  // per device

// caller holds g_pin_mu
static void reclaim_completed_slots() {
  for (size_t i = 0; i < g_pin_pending.size();) {
    if (cudaEventQuery(g_pin_pending[i].ev) == cudaSuccess) {
      g_pin_free.push_back(g_pin_pending[i].slot);
      g_free_events[g_pin_pending[i].dev].push_back(g_pin_pending[i].ev);
      g_pin_pending[i] = g_pin_pending.back();
      g_pin_pending.pop_back();
    } else {
      i++;
    }
  }
}

int pinned_acquire(void **p) {
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    if (g_pin_free.empty()) reclaim_completed_slots();
    if (!g_pin_free.empty()) {
      *p = g_pin_free.back();
      g_pin_free.pop_back();
      return GM_OK;
    }
  }
  cudaError_t e = cudaMallocHost(p, PINNED_SLOT_BYTES);
  if (e != cudaSuccess) return record_error(e, "cudaMallocHost(tail slot)");
  return GM_OK;
}

void pinned_release(void *p) {
  std::lock_guard<std::mutex> lk(g_pin_mu);
  g_pin_free.push_back(p);
}

// The slot returns to the pool once the work enqueued on s so far has run.
int enqueue_pinned_release(cudaStream_t s, void *slot) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return record_error(e, "cudaGetDevice");
  cudaEvent_t ev = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    auto &fe = g_free_events[dev];
    if (!fe.empty()) {
      ev = fe.back();
      fe.pop_back();
    }
  }
  if (ev == nullptr) {
    e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    // without an event the slot stays with the stream's pending work: leak it
    // rather than hand it out again while a copy may still use it
    if (e != cudaSuccess) return record_error(e, "cudaEventCreate(slot)");
  }
  e = cudaEventRecord(ev, s);
  if (e != cudaSuccess) return record_error(e, "cudaEventRecord(slot)");
  std::lock_guard<std::mutex> lk(g_pin_mu);
  g_pin_pending.push_back(PendingSlot{slot, ev, dev});
  return GM_OK;
}

int device_sm_count(int dev, int *sms) {
  DeviceState *st;
  int rc = device_state(dev, &st);
  if (rc) return rc;
  *sms = st->sms;
  return GM_OK;
}

int select_device(uint32_t gpu_index) {
  int count = 0;
  GM_CHECK(cudaGetDeviceCount(&count));
  if ((int)gpu_index >= count) {
    set_last_error("gpu_index out of range");
    return GM_ERR_ARG;
  }
  GM_CHECK(cudaSetDevice((int)gpu_index));
  return GM_OK;
}

int pool_alloc(int dev, cudaStream_t s, size_t bytes, void **ptr) {
  DeviceState *st;
  int rc = device_state(dev, &st);
  if (rc) return rc;
  cudaError_t e = cudaMallocFromPoolAsync(ptr, bytes, st->pool, s);
  if (e != cudaSuccess) {
    record_error(e, "cudaMallocFromPoolAsync");
    return GM_ERR_ALLOC;
  }
  return GM_OK;
}

// ---------------------------------------------------------------------------
// scratch blocks (msm_engine.h)
// ---------------------------------------------------------------------------
struct ScratchBlock {
  char *p = nullptr;
  size_t bytes = 0;
  cudaEvent_t done = nullptr;  // after the block's last use
  cudaStream_t last = nullptr;
  uint64_t turn = 0;  // of the last use
};
struct ScratchArena {
  std::mutex mu;
  ScratchBlock blocks[SCRATCH_BLOCKS];
  uint64_t turns = 0;
};

static ScratchArena &scratch_arena(int dev) {
  static std::mutex mu;
  static std::map<int, ScratchArena> arenas;  // nodes stay where they are
  std::lock_guard<std::mutex> lk(mu);
  return arenas[dev];
}

bool device_room(size_t bytes) {
  // also while this thread captures a stream, whose work the question is no part of
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  size_t free_bytes = 0, all = 0;
  const cudaError_t e = cudaMemGetInfo(&free_bytes, &all);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e == cudaSuccess) return free_bytes / 2 >= bytes;
  cudaGetLastError();
  return false;
}

static void scratch_drop(ScratchBlock &b) {
  if (b.p == nullptr) return;
  cudaEventSynchronize(b.done);
  cudaFree(b.p);
  cudaEventDestroy(b.done);
  b = ScratchBlock();
}

// four sizes from one power of two to the next: calls of slightly different sizes share a block
size_t scratch_block_bytes(size_t bytes) {
  size_t step = size_t(16) << 20;
  while (8 * step < bytes) step *= 2;
  return (bytes + step - 1) / step * step;
}

static bool scratch_create(ScratchBlock &b, size_t bytes) {
  const size_t up = scratch_block_bytes(bytes);
  if (!device_room(up)) return false;
  if (cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming) == cudaSuccess) {
    if (cudaMalloc(&b.p, up) == cudaSuccess) {
      b.bytes = up;
      return true;
    }
    cudaEventDestroy(b.done);
  }
  cudaGetLastError();
  b = ScratchBlock();
  return false;
}

char *ScratchLease::acquire(int dev, cudaStream_t s, size_t bytes) {
  release();
  dev_ = dev;
  s_ = s;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    void *p = nullptr;
    if (!device_room(bytes) || pool_alloc(dev, s, bytes, &p) != GM_OK) {
      cudaGetLastError();
      return nullptr;
    }
    return captured_ = static_cast<char *>(p);
  }
  ScratchArena &a = scratch_arena(dev);
  std::unique_lock<std::mutex> lk(a.mu);
  // the stream's own last block, an idle one, a new one, the one in use for longest, a new one in place of a smaller
  ScratchBlock *own = nullptr, *idle = nullptr, *used = nullptr, *empty = nullptr, *small = nullptr;
  for (ScratchBlock &b : a.blocks) {
    if (b.p == nullptr) {
      empty = &b;
    } else if (b.bytes < bytes) {
      if ((!small || b.bytes < small->bytes) && cudaEventQuery(b.done) == cudaSuccess) small = &b;
    } else if (b.last == s) {
      own = &b;
    } else if (cudaEventQuery(b.done) == cudaSuccess) {
      idle = &b;
    } else if (!used || b.turn < used->turn) {
      used = &b;
    }
  }
  ScratchBlock *take = own ? own : idle;
  if (!take && empty && scratch_create(*empty, bytes)) take = empty;
  if (!take) take = used;
  if (!take && small) {
    scratch_drop(*small);
    if (scratch_create(*small, bytes)) take = small;
  }
  cudaGetLastError();  // a query's "not ready"
  if (!take || cudaStreamWaitEvent(s, take->done, 0) != cudaSuccess) return nullptr;
  take->last = s;
  take->turn = ++a.turns;
  lk.release();  // until release()
  block_ = take;
  return take->p;
}

void ScratchLease::release() {
  if (captured_) cudaFreeAsync(captured_, s_);
  captured_ = nullptr;
  if (!block_) return;
  if (cudaEventRecord(block_->done, s_) != cudaSuccess) cudaStreamSynchronize(s_);
  block_ = nullptr;
  scratch_arena(dev_).mu.unlock();
}

int trim_memory(int dev) {
  GM_CHECK(cudaDeviceSynchronize());
  {
    ScratchArena &a = scratch_arena(dev);
    std::lock_guard<std::mutex> lk(a.mu);
    for (ScratchBlock &b : a.blocks) scratch_drop(b);
  }
  DeviceState *st;
  const int rc = device_state(dev, &st);
  if (rc) return rc;
  GM_CHECK(cudaMemPoolTrimTo(st->pool, 0));
  GM_CHECK(cudaDeviceGraphMemTrim(dev));  // of captured calls whose graphs are gone
  return GM_OK;
}

// ---------------------------------------------------------------------------
// window selection (cost model in multiplication units)
//   accumulation: 10 per (point, non-zero window) (madd 8M+2S), 7 where rounds
//                 of affine additions run first (about 3 M entries up)
//   reduction:    two full additions of 14 mults per bucket and the upper
//                 levels: 38; 48 (G1) and 60 (G2) against the cheaper entries
//   combine:      c doublings (9 mults) per window in one chain: weighted
//                 by the serial latency against a wave of the whole GPU.
// B200, best width measured (the model's where it differs): G1 2^18 12, 400000
// 12, 600000 15, 2^20 15, 2^21 15; G2 130000 12, 2^18 12, 2^19 14; with 10 and 38
// throughout the model took 15 for G1 2^18 (4.12 against 3.87 ms), 16 for 2^20
// (11.3 / 10.9), 15 for G2 2^18 (10.5 / 9.5).
// ---------------------------------------------------------------------------
static int windows_for(int c, int limbs) { return (64 * limbs) / c + 1; }

int default_window(int group, int64_t n, int limbs) {
  if (n <= 0) return 4;
  const int sbits = std::min(64 * limbs, 299);  // scalars below r have 299 significant bits
  const bool rounds = (double)n * sbits >= 3e6 * 12;
  double best = 1e300;
  int best_c = 4;
  for (int c = 3; c <= 18; c++) {
    const int W = windows_for(c, limbs);
    const int Weff = sbits / c + 1;
    const double acc = (rounds ? 7.0 : 10.0) * (double)n * Weff;
    const double red = (rounds ? (group == 1 ? 48.0 : 60.0) : 38.0) * (double)W * std::ldexp(1.0, c - 1);
    const double tail = 9.0 * c * Weff * 2000.0;
    // Hot buckets: a top window of few bits puts all n of its entries into a
    // handful of buckets, and a full top window (c bits, so digits above
    // 2^(c-1)) carries into one more window whose single bucket gets about
    // n/2 entries; both mean long fix-up runs and contended sort counters
    // (G1 2^17: c = 11, 2 top bits, 0.32 ms more fix-up and sort than c = 12;
    // G2 2^16: c = 11 0.63 ms, c = 13 (full top window) 0.31 ms more).
    const int top_bits = sbits - c * ((sbits + c - 1) / c - 1);
    const double hot = (top_bits <= 3 || top_bits >= c) ? 40.0 * (double)n : top_bits <= 6 ? 20.0 * (double)n : 0.0;
    const double cost = acc + red + tail + hot;
    if (cost < best) {
      best = cost;
      best_c = c;
    }
  }
  return best_c;
}

}  // namespace gm
