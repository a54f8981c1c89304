// Internal interface between the C-ABI layer (capi.cu, field_kernels.cu) and
// the MSM engine (msm.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace gm {

enum {
  GM_OK = 0,
  GM_ERR_ARG = -1,
  GM_ERR_STREAM = -2,
  GM_ERR_ALLOC = -3,
  GM_ERR_CUDA = -4,
  GM_ERR_CHECK = -5,
};

int record_error(cudaError_t e, const char *where);
const char *last_error();
int select_device(uint32_t gpu_index);
int device_sm_count(int dev, int *sms);
void set_last_error(const char *msg);

// phase profiling: when enabled, msm_launch records a CUDA event on the
// launching stream at every phase boundary; profile_collect synchronises
// them and returns per-phase milliseconds.
void profile_enable(bool on);
bool profile_enabled();
void profile_mark(cudaStream_t s, const char *name);
void profile_end_call();
int profile_collect(char *names, int names_len, float *ms, int max);
// Pinned host slots of PINNED_SLOT_BYTES, recycled; enqueue_pinned_release
// hands a slot back once the stream reaches that point.
constexpr size_t PINNED_SLOT_BYTES = 128 * 1024;
int pinned_acquire(void **p);
void pinned_release(void *p);
int enqueue_pinned_release(cudaStream_t s, void *slot);
// kernel launches issued by this host thread since the last reset
void count_launches(int k);
int64_t launches_and_reset();
int pool_alloc(int dev, cudaStream_t s, size_t bytes, void **ptr);
int default_window(int group, int64_t n, int limbs);

// Device memory that one call's kernels use for a part of their run and that
// later calls, on any stream, take over: the scratch of the affine rounds.
//
// A device keeps up to SCRATCH_BLOCKS blocks.  acquire orders the stream after
// the block's last use and holds it for the calling thread, which enqueues its
// kernels and then calls release; the host waits only while another thread
// enqueues.  A call takes a block that is idle or was last used on its own
// stream, or a new one; only with SCRATCH_BLOCKS calls in flight does it take
// its turn behind one of them, so that the memory kept is bounded whatever the
// number of streams.  (The rounds fill the GPU: three streams of G1 2^20 points
// take 10.1 ms a call with three blocks and with one.)  A block comes from cudaMalloc:
// 3 GB take 0.8 ms where a stream-ordered pool maps them in 18 ms, which a
// process's first call at a size would pay (B200, first G1 2^20 call 31 to 37 ->
// 17 ms).  While s is being captured the memory is a graph allocation of its
// own.  acquire returns null, and the caller does without, where the device
// does not have twice the bytes free.
constexpr int SCRATCH_BLOCKS = 4;
struct ScratchBlock;
class ScratchLease {
 public:
  ScratchLease() = default;
  ScratchLease(const ScratchLease &) = delete;
  ScratchLease &operator=(const ScratchLease &) = delete;
  ~ScratchLease() { release(); }
  char *acquire(int dev, cudaStream_t s, size_t bytes);
  void release();

 private:
  int dev_ = 0;
  cudaStream_t s_ = nullptr;
  char *captured_ = nullptr;       // graph allocation
  ScratchBlock *block_ = nullptr;  // held, with its device's lock
};
// Size of a block for that many bytes.
size_t scratch_block_bytes(size_t bytes);
// Whether the device has twice these bytes free.
bool device_room(size_t bytes);
// Gives the kept blocks and the pool's unused memory back to the device.
int trim_memory(int dev);

// Window sums handed to a synchronous caller in place of the device
// combination: the MSM copies its W window sums (XYZZ, device layout) to
// `host` (pinned, `cap` bytes), sets W and c and writes no result; the caller
// combines them (gm_host::horner_to_proj) after synchronising the stream.
struct TailHandoff {
  void *host = nullptr;
  size_t cap = 0;
  int W = 0, c = 0;
};

// Full MSM pipeline on `s`.  Either `bases` (packed records) or `ref_points`
// (reference-layout affine points; converted to Montgomery when to_mont) is
// given.  Writes the result (reference layout; projective, or affine) to out.  When
// err_out is non-null it receives the device consistency flag (0 = ok).
// bases_ready (optional): an event the stream waits for after the sort,
// before the bases are first read (the sort reads only the scalars).
// handoff (optional, not while capturing): the window sums go to the caller
// instead of a result in out.
template <class F>
int msm_launch(cudaStream_t s, int dev, const uint4 *bases, const uint64_t *ref_points, int to_mont,
               const uint64_t *scalars, int limbs, int64_t n, uint64_t *out, int c_override, uint32_t *err_out,
               cudaEvent_t bases_ready = nullptr, TailHandoff *handoff = nullptr, bool affine = false);

}  // namespace gm
