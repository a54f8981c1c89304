// Bucket accumulation of large MSMs by rounds of affine additions.
//
// A round adds the points of every bucket in pairs: a bucket of s points
// leaves ceil(s / 2).  All pairs of a round are independent, so a thread takes
// a run of them and shares one field inversion among up to AFF_BATCH
// (Montgomery's trick): an addition costs 3 products for the inversion's
// share, 2 products and a square, against 8 products and 2 squares of the XYZZ
// mixed addition of k_accumulate.  After `rounds` rounds (AffLayout::plan:
// until a bucket of ordinary size is down to one point) k_accumulate runs over
// what is left, which is one point of most buckets and the rest of the few
// that are much larger, so those need no rule of their own here.
//
// Bound: the multiplier, as for k_accumulate (a round moves 640 bytes an
// addition, 1.5 TB/s).  B200, G1 2^20 at c = 16 (19.5 M entries, 28 to a
// bucket): 0.42 ns an addition in the first rounds against 0.55 ns in
// k_accumulate; accumulation in all 11.1 -> 8.8 ms, G2 2^18 8.7 -> 7.0 ms (at
// c = 15).  With the widths now chosen (15, 12): 8.0 + 0.8 and 6.4 + 1.4 ms, the
// multiplier 70-75 % busy in the rounds.  Three blocks of 128 threads per SM
// (G1): two measured 9.14 ms against 8.79 for six rounds, four 9.00 (the
// code of product, square, inversion and loops then outgrows the instruction
// cache).
//
// The points of a round lie in bucket order: round r's offsets are the prefix
// sums of ceil(s / 2^r), all computed at once from the sorted entries'
// offsets.  A round reads records by index (the first one through the sorted
// entries, with their signs) and writes records; x = y = 0 is infinity.  Keys
// (buckets) are processed in chunks of whole groups so that the two buffers
// the rounds alternate between stay within AFF_SCRATCH bytes; a single group may
// take twice that (MSMs of 2^25 points), and a larger one runs without rounds.
#pragma once
#include <algorithm>
#include <vector>

#include "msm_kernels.cuh"

namespace gm {

constexpr int AFF_THREADS = 128;
constexpr int AFF_BATCH = 64;       // additions that share an inversion, at most
constexpr int AFF_MIN = 16;         // outputs of a thread, at least (a shorter run spends more on its inversion)
constexpr int AFF_MAX_ROUNDS = 8;
// Outputs per thread of the last round, at least, for both groups.  Flat from 10
// to 16 for single MSMs; not measured below 10 or for batches.  With 10 / 16 / 24
// / 40: G1 2^20 11.52 / 11.41 / 11.38 / 11.40 ms, G1 2^18 4.23 / 4.18 / 4.18 /
// 4.25, G1 200000 3.41 / 3.34 / 3.46 / 3.46, G2 130000 6.18 / 6.13 / 6.48 / 6.47,
// G2 65536 4.33 / 4.27 / 4.60 / 4.60 (without rounds: 13.66, 4.56, 3.77, 7.23, 4.60).
constexpr int AFF_LAST = 16;
// The two buffers' bytes in all: a chunk's last round and every round's last
// blocks leave the GPU partly idle, so fewer chunks are better.  Measured with
// 0.5 / 1 / 3 / 6 / 12 GiB: G1 2^20 12.3 / 11.3 / 10.8 (one chunk), G1 2^21 26.0 /
// 21.2 / 20.1 / 19.5 / 19.5, G2 2^20 42.0 / 32.2 / 29.2 / 28.9 / 28.9, 512 MSMs of
// 6 M points 122.6 / 106.9 / 97.3 / 96.6 / 95.7 ms.
constexpr size_t AFF_SCRATCH = size_t(3) << 30;
template <class F>
constexpr int AFF_BLOCKS = sizeof(typename F::T) == sizeof(fp_t) ? 3 : 2;  // resident blocks per SM

// Out-of-line products of a round (both the product and the square: the loop
// holds one body of each)
template <class F>
struct AffPolicy;
template <>
struct AffPolicy<Fp> {
  using type = FpOut;
};
template <>
struct AffPolicy<Fp2> {
  using type = Fp2Call;
};

// ---------------------------------------------------------------------------
// Offsets of every round: off[r][k] = sum of ceil(s / 2^(r+1)) below k, from
// the offsets off0 of the sorted entries.  One block row per round.
// ---------------------------------------------------------------------------
GM_DEVI uint32_t aff_size(const uint32_t *__restrict__ off0, int64_t k, int64_t K, int r) {
  if (k >= K) return 0u;
  const uint32_t s = __ldg(off0 + k + 1) - __ldg(off0 + k);
  return (s >> r) + ((s & ((1u << r) - 1u)) ? 1u : 0u);
}
static __global__ void k_aff_blocksum(const uint32_t *__restrict__ off0, int64_t K, uint32_t *__restrict__ bsum) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  const int r = blockIdx.y + 1;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; k++) s += aff_size(off0, base + k, K, r);
  uint32_t total;
  block_exclusive_scan(s, total);
  if (threadIdx.x == 0) bsum[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = total;
}
static __global__ void k_aff_top(uint32_t *__restrict__ bsum, int nb) {
  bsum += (int64_t)blockIdx.x * nb;
  uint32_t running = 0;
  for (int base = 0; base < nb; base += SCAN_TILE) {
    const int i0 = base + threadIdx.x * SCAN_PER_THREAD;
    uint32_t v[SCAN_PER_THREAD], s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; k++) {
      v[k] = (i0 + k < nb) ? bsum[i0 + k] : 0;
      s += v[k];
    }
    uint32_t total;
    uint32_t ex = block_exclusive_scan(s, total) + running;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; k++) {
      if (i0 + k < nb) bsum[i0 + k] = ex;
      ex += v[k];
    }
    running += total;
    __syncthreads();
  }
}
static __global__ void k_aff_offsets(const uint32_t *__restrict__ off0, int64_t K, const uint32_t *__restrict__ bsum,
                                     uint32_t *__restrict__ off, int64_t stride) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  const int r = blockIdx.y + 1;
  off += (int64_t)blockIdx.y * stride;
  uint32_t v[SCAN_PER_THREAD], s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; k++) {
    v[k] = aff_size(off0, base + k, K, r);
    s += v[k];
  }
  uint32_t total;
  uint32_t ex = block_exclusive_scan(s, total) + bsum[(int64_t)blockIdx.y * gridDim.x + blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; k++) {
    if (base + k < K) off[base + k] = ex;
    if (base + k == K - 1) off[K] = ex + v[k];
    ex += v[k];
  }
}

// ---------------------------------------------------------------------------
// One round
// ---------------------------------------------------------------------------

// x (y) of a packed record
template <class F>
GM_DEVI void load_coord(typename F::T &v, const uint4 *rec, bool y) {
  constexpr int L = F::LIMBS;  // 14 or 28 words: y starts at a 16-byte boundary for Fp2, 8 bytes past one for Fp
  if constexpr (L % 4 == 0) {
    const uint4 *p = rec + (y ? L / 4 : 0);
#pragma unroll
    for (int q = 0; q < L / 4; q++) {
      const uint4 w = __ldg(p + q);
      limb_ref<F>(v, 4 * q) = w.x;
      limb_ref<F>(v, 4 * q + 1) = w.y;
      limb_ref<F>(v, 4 * q + 2) = w.z;
      limb_ref<F>(v, 4 * q + 3) = w.w;
    }
  } else {
    const uint2 *p = reinterpret_cast<const uint2 *>(rec) + (y ? L / 2 : 0);
#pragma unroll
    for (int q = 0; q < L / 2; q++) {
      const uint2 w = __ldg(p + q);
      limb_ref<F>(v, 2 * q) = w.x;
      limb_ref<F>(v, 2 * q + 1) = w.y;
    }
  }
}

// Where an output's inputs lie: record index << 1, and the sign to apply to y
// in bit 0 (the sorted entries of the first round have this form).
struct AffPair {
  uint32_t p, q;
  bool pair;  // q is there
};

// Walk over a chunk's outputs: bucket k holds outputs [ob, oe) of inputs [ib, ie).
template <bool FIRST>
struct AffWalk {
  const uint32_t *entries, *off_in, *off_out;
  uint32_t in0;
  int64_t k0, k1;  // the chunk's buckets
  int64_t k;
  uint32_t ob, oe, ib, ie;
  GM_DEVI void start(int64_t k_) {
    k = k_;
    ob = __ldg(off_out + k);
    oe = __ldg(off_out + k + 1);
    ib = __ldg(off_in + k);
    ie = __ldg(off_in + k + 1);
  }
  GM_DEVI AffPair at(uint32_t j) const {
    const uint32_t a = ib + 2 * (j - ob);
    AffPair r;
    r.pair = a + 1 < ie;
    if (FIRST) {
      r.p = __ldg(entries + a);
      r.q = r.pair ? __ldg(entries + a + 1) : 0u;
    } else {
      r.p = (a - in0) << 1;
      r.q = r.p + 2;
    }
    return r;
  }
  GM_DEVI AffPair forward(uint32_t j) {
    for (int s = 0; j >= oe; s++) {
      if (s == 4) {  // a run of empty buckets
        start(k + bucket_of(off_out + k, k1 - k, j));
        break;
      }
      k++;
      ob = oe;
      oe = __ldg(off_out + k + 1);
      ib = ie;
      ie = __ldg(off_in + k + 1);
    }
    return at(j);
  }
  GM_DEVI AffPair backward(uint32_t j) {
    for (int s = 0; j < ob; s++) {
      if (s == 4) {
        start(k0 + bucket_of(off_out + k0, k - k0, j));
        break;
      }
      k--;
      oe = ob;
      ob = __ldg(off_out + k);
      ie = ib;
      ib = __ldg(off_in + k);
    }
    return at(j);
  }
};

// Shared-memory stage of one thread ([chunk][thread] uint4): the two points
// of a pair and its prefix product, brought in with cp.async while a product
// of the same or the previous addition runs, so one slot is enough.
template <class F>
struct AffStage {
  static constexpr int XC = (F::LIMBS + 3) / 4;  // chunks of an element (Fp: and the first 2 words of y)
  static constexpr int RC = F::LIMBS / 2;        // chunks of a point
  static constexpr int CH = 2 * RC + XC;         // P, Q, prefix
  static constexpr int BYTES = CH * AFF_THREADS * 16;
};

template <class F>
GM_DEVI typename F::T stage_get(const uint4 (*c)[AFF_THREADS], int tid, int first_word) {
  typename F::T r;
#pragma unroll
  for (int k = 0; k < F::LIMBS; k++) {
    const int i = first_word + k;
    const uint4 v = c[i >> 2][tid];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    limb_ref<F>(r, k) = w[i & 3];
  }
  return r;
}

template <class F>
GM_DEVI void store_point(uint4 *dst, typename F::T &x, typename F::T &y) {
  constexpr int L = F::LIMBS;
  uint32_t w[2 * L];
#pragma unroll
  for (int k = 0; k < L; k++) {
    w[k] = limb_ref<F>(x, k);
    w[L + k] = limb_ref<F>(y, k);
  }
#pragma unroll
  for (int q = 0; q < L / 2; q++) dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}

// Outputs off_out[k0] .. off_out[k1] of one chunk of keys.  in: records (the
// bases in the first round, with the sorted entries; else the previous round's
// records of this chunk).  out receives this chunk's records, from its first
// one on (local_out) or at their index over all keys.  prefix: AFF_BATCH
// elements per thread of the grid, interleaved by 16-byte chunks.
template <class F, bool FIRST>
__global__ void __launch_bounds__(AFF_THREADS, AFF_BLOCKS<F>)
    k_affine_round(const uint4 *__restrict__ in, const uint32_t *__restrict__ entries,
                   const uint32_t *__restrict__ off_in, const uint32_t *__restrict__ off_out, int64_t k0, int64_t k1,
                   uint4 *__restrict__ out, bool local_out, uint4 *__restrict__ prefix) {
  using A = typename AffPolicy<F>::type;
  using T = typename F::T;
  using S = AffStage<F>;
  constexpr int L = F::LIMBS, U4 = Rec<F>::U4;
  extern __shared__ uint4 stage_mem[];
  auto stage = reinterpret_cast<uint4(*)[AFF_THREADS]>(stage_mem);
  const uint4(*const P)[AFF_THREADS] = stage, (*const Q)[AFF_THREADS] = stage + S::RC, (*const R)[AFF_THREADS] = stage + 2 * S::RC;
  const int tid = threadIdx.x;
  const uint32_t o0 = __ldg(off_out + k0), o1 = __ldg(off_out + k1);
  const uint32_t nthr = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + tid;
  const uint32_t M = o1 - o0;
  const uint32_t chunk = max((M + nthr - 1) / nthr, (uint32_t)AFF_MIN);
  const uint64_t start64 = (uint64_t)o0 + (uint64_t)t * chunk;
  if (start64 >= o1) return;
  const uint32_t end = (uint32_t)min(start64 + chunk, (uint64_t)o1);
  AffWalk<FIRST> walk{entries, off_in, off_out, FIRST ? 0u : __ldg(off_in + k0), k0, k1};
  walk.start(k0 + bucket_of(off_out + k0, k1 - k0, (uint32_t)start64));
  out -= (size_t)(local_out ? o0 : 0u) * U4;

  auto rec = [&](uint32_t e) { return in + (size_t)(e >> 1) * U4; };
  auto coord_y = [&](uint32_t e) {  // from memory, with the entry's sign
    T y;
    load_coord<F>(y, rec(e), true);
    return FIRST && (e & 1u) ? F::neg(y) : y;
  };
  auto pre = [&](int i, int q) -> uint4 * { return prefix + ((size_t)i * S::XC + q) * nthr + t; };

  // equal batches
  const uint32_t nbatch = (end - (uint32_t)start64 + AFF_BATCH - 1) / AFF_BATCH;
  const uint32_t bsize = (end - (uint32_t)start64 + nbatch - 1) / nbatch;
  for (uint32_t s0 = (uint32_t)start64; s0 < end; s0 += bsize) {
    const int cnt = (int)min(end - s0, bsize);
    uint64_t m_mul = 0, m_dbl = 0, m_b = 0, m_inf = 0;  // additions, doublings among them, copies of q, infinity
    T run;
    AffPair c0, c1 = walk.forward(s0);
    auto stage_x = [&](const AffPair &c) {
      if (c.pair) {
#pragma unroll
        for (int q = 0; q < S::XC; q++) {
          cp_async16(&stage[q][tid], rec(c.p) + q);
          cp_async16(&stage[S::RC + q][tid], rec(c.q) + q);
        }
      }
      cp_async_commit();
    };
    stage_x(c1);
#pragma unroll 1
    for (int i = 0; i < cnt; i++) {
      c0 = c1;
      if (i + 1 < cnt) c1 = walk.forward(s0 + i + 1);
      cp_async_wait<0>();
      const T x1 = stage_get<F>(P, tid, 0);
      T d = stage_get<F>(Q, tid, 0);
      if (i + 1 < cnt) stage_x(c1);  // the next x's arrive during this product
      if (!c0.pair) continue;        // the odd point out
      bool add = true;
      const bool z1 = F::is_zero_raw(x1), z2 = F::is_zero_raw(d);
      d = F::sub(d, x1);
      const bool e = F::is_zero_raw(d);
      if (z1 || z2 || e) {
        const T y1 = coord_y(c0.p), y2 = coord_y(c0.q);
        const bool i1 = z1 && F::is_zero_raw(y1), i2 = z2 && F::is_zero_raw(y2);
        if (i1 || i2) {
          if (i1) m_b |= 1ull << i;  // infinity + q, also when q is infinity
          add = false;
        } else if (e) {
          if (F::eq(y1, y2) && !F::is_zero_raw(y1)) {
            d = F::dbl(y1);
            m_dbl |= 1ull << i;
          } else {
            m_inf |= 1ull << i;
            add = false;
          }
        }
      }
      if (add) {
        if (m_mul) {
#pragma unroll
          for (int q = 0; q < S::XC; q++) {
            uint4 w;
            w.x = limb_ref<F>(run, 4 * q);
            w.y = limb_ref<F>(run, 4 * q + 1);
            w.z = 4 * q + 2 < L ? limb_ref<F>(run, 4 * q + 2 < L ? 4 * q + 2 : 0) : 0u;
            w.w = 4 * q + 3 < L ? limb_ref<F>(run, 4 * q + 3 < L ? 4 * q + 3 : 0) : 0u;
            *pre(i, q) = w;
          }
          run = A::mul(run, d);
        } else {
          run = d;
        }
        m_mul |= 1ull << i;
      }
    }
    T inv;
    if (m_mul) inv = A::inv(run);
    __threadfence();  // this thread's prefix products, which come back through cp.async

    const AffWalk<FIRST> ahead = walk;  // where the next batch goes on
    auto stage_prefix = [&](int i) {
      if (i >= 0 && (m_mul >> i & 1) && (m_mul & ((1ull << i) - 1))) {
#pragma unroll
        for (int w = 0; w < S::XC; w++) cp_async16(&stage[2 * S::RC + w][tid], pre(i, w));
      }
      cp_async_commit();
    };
    stage_prefix(cnt - 1);
    c1 = walk.backward(s0 + cnt - 1);
#pragma unroll 1
    for (int i = cnt - 1; i >= 0; i--) {
      const uint64_t bit = 1ull << i;
      c0 = c1;
      if (m_mul & bit) {
        const uint4 *p = rec(c0.p), *q = rec(c0.q);
#pragma unroll
        for (int w = 0; w < S::RC; w++) {
          cp_async16(&stage[w][tid], p + w);
          cp_async16(&stage[S::RC + w][tid], q + w);
        }
      }
      cp_async_commit();
      if (i > 0) c1 = walk.backward(s0 + i - 1);
      uint4 *dst = out + (size_t)(s0 + i) * U4;
      auto y_of = [&](const uint4(*c)[AFF_THREADS], uint32_t e) -> T {
        const T y = stage_get<F>(c, tid, L);
        return FIRST && (e & 1u) ? F::neg(y) : y;
      };
      if (m_mul & bit) {
        const bool dbl = (m_dbl & bit) != 0;
        T lam = inv;
        cp_async_wait<1>();  // the prefix product
        if (m_mul & (bit - 1)) {  // not the batch's first addition
          lam = stage_get<F>(R, tid, 0);
          stage_prefix(i - 1);
          lam = A::mul(lam, inv);
          cp_async_wait<1>();  // the points
          inv = A::mul(inv, dbl ? F::dbl(y_of(P, c0.p)) : F::sub(stage_get<F>(Q, tid, 0), stage_get<F>(P, tid, 0)));
        } else {
          cp_async_wait<0>();
        }
        T num;
        if (dbl) {
          const T x = stage_get<F>(P, tid, 0);
          const T xx = A::mul(x, x);
          num = F::add(F::dbl(xx), xx);
        } else {
          num = F::sub(y_of(Q, c0.q), y_of(P, c0.p));
        }
        lam = A::mul(lam, num);
        T x3 = A::sqr(lam);
        const T x1 = stage_get<F>(P, tid, 0);
        x3 = F::sub(F::sub(x3, x1), stage_get<F>(Q, tid, 0));
        T y3 = F::sub(A::mul(lam, F::sub(x1, x3)), y_of(P, c0.p));
        store_point<F>(dst, x3, y3);
      } else if (m_inf & bit) {
        T z = F::zero();
        store_point<F>(dst, z, z);
        stage_prefix(i - 1);
      } else {
        stage_prefix(i - 1);
        const uint32_t e = (m_b & bit) ? c0.q : c0.p;
        T x, y = coord_y(e);
        load_coord<F>(x, rec(e), false);
        store_point<F>(dst, x, y);
      }
    }
    walk = ahead;
    cp_async_wait<0>();  // the next batch reuses this thread's stage
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct AffLayout {
  int rounds = 0;  // 0: the accumulation runs without affine rounds
  int64_t K = 0;
  struct Chunk {
    int64_t k0, k1;
  };
  std::vector<Chunk> chunks;
  // own memory: offsets of every round, block sums, the points left over
  size_t bytes = 0, o_off = 0, o_bsum = 0, o_fin = 0;
  // scratch of the rounds (accumulations that run one after another can share it)
  size_t scratch = 0, s_buf1 = 0, s_prefix = 0;
  unsigned grid = 0;

  // what the rounds leave in the own memory m: points in bucket order, and their offsets
  const uint32_t *final_offsets(const char *m) const {
    return (const uint32_t *)(m + o_off) + (int64_t)(rounds - 1) * (K + 1);
  }
  const uint4 *final_points(const char *m) const { return (const uint4 *)(m + o_fin); }

  // sizes: points of the MSMs; each has `groups` key groups (windows, or 1
  // over a fixed-base table) of B keys, every group at most per_point entries
  // per point.  K keys in all.
  //
  // A round pays while its threads have enough outputs to share an inversion
  // and buckets still hold two points or more.
  template <class F, class Carver>
  void plan(const int64_t *sizes, int count, int groups, int per_point, int B, int sms) {
    Carver cv;
    int64_t E = 0;
    for (int i = 0; i < count; i++) E += sizes[i] * per_point * groups;
    K = (int64_t)count * groups * B;
    const double avg = (double)E / (double)K;
    constexpr size_t REC = Rec<F>::U4 * sizeof(uint4);
    grid = (unsigned)(sms * AFF_BLOCKS<F>);
    const int64_t threads = (int64_t)grid * AFF_THREADS;
    int R = 0;
    while (R < AFF_MAX_ROUNDS && (E >> (R + 1)) >= AFF_LAST * threads && (2 << R) <= avg) R++;
    if (R == 0) return;
    // outputs of a chunk of e entries and k keys after r + 1 rounds
    auto outputs = [](int64_t e, int64_t k, int r) {
      return std::min(e, ((e + k * ((int64_t(2) << r) - 1)) >> (r + 1)) + 1);
    };
    // chunks of whole groups, the buffers of the first two rounds within the scratch
    int64_t e = 0, k = 0, b0 = 0, b1 = 0, kbase = 0;
    std::vector<Chunk> ch;
    auto close = [&] {
      if (k == 0) return;
      b0 = std::max(b0, outputs(e, k, 0));
      b1 = std::max(b1, outputs(e, k, 1));
      ch.push_back(Chunk{kbase, kbase + k});
      kbase += k;
      e = k = 0;
    };
    for (int i = 0; i < count; i++)
      for (int w = 0; w < groups; w++) {
        const int64_t ge = sizes[i] * per_point;
        const auto need = [&](int64_t ee, int64_t kk) { return (size_t)(outputs(ee, kk, 0) + outputs(ee, kk, 1)) * REC; };
        if (need(ge, B) > 2 * AFF_SCRATCH) return;  // a group too large for the buffers: no rounds
        if (k > 0 && need(e + ge, k + B) > AFF_SCRATCH) close();
        e += ge;
        k += B;
      }
    close();
    rounds = R;
    chunks = std::move(ch);
    const int64_t nb = (K + SCAN_TILE - 1) / SCAN_TILE;
    o_off = cv.template take<uint32_t>((size_t)(R * (K + 1)));
    o_bsum = cv.template take<uint32_t>((size_t)(R * nb));
    o_fin = cv.template take<uint4>((size_t)outputs(E, K, R - 1) * Rec<F>::U4);
    bytes = cv.off;
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    s_buf1 = up((size_t)b0 * REC);
    s_prefix = s_buf1 + (R > 1 ? up((size_t)b1 * REC) : 0);
    scratch = s_prefix + (size_t)grid * AFF_THREADS * AFF_BATCH * AffStage<F>::XC * sizeof(uint4);
  }
};

// Enqueues the rounds on s, in the layout's own memory m and the scratch.
template <class F>
cudaError_t aff_launch(cudaStream_t s, const AffLayout &lay, char *m, char *scratch, const uint4 *bases,
                       const uint32_t *entries, const uint32_t *off0, int *launches) {
  const int R = lay.rounds;
  const int64_t K = lay.K;
  for (const void *fn : {(const void *)k_affine_round<F, true>, (const void *)k_affine_round<F, false>}) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, AffStage<F>::BYTES);
    if (e != cudaSuccess) return e;
  }
  const unsigned nb = (unsigned)((K + SCAN_TILE - 1) / SCAN_TILE);
  auto *off = (uint32_t *)(m + lay.o_off);
  auto *bsum = (uint32_t *)(m + lay.o_bsum);
  k_aff_blocksum<<<dim3(nb, R), SCAN_THREADS, 0, s>>>(off0, K, bsum);
  k_aff_top<<<R, SCAN_THREADS, 0, s>>>(bsum, (int)nb);
  k_aff_offsets<<<dim3(nb, R), SCAN_THREADS, 0, s>>>(off0, K, bsum, off, K + 1);
  *launches += 3;
  uint4 *buf[2] = {(uint4 *)scratch, (uint4 *)(scratch + lay.s_buf1)};
  auto *prefix = (uint4 *)(scratch + lay.s_prefix);
  for (const auto &c : lay.chunks) {
    for (int r = 0; r < R; r++) {
      const uint32_t *off_out = off + (int64_t)r * (K + 1);
      uint4 *out = r == R - 1 ? (uint4 *)(m + lay.o_fin) : buf[r & 1];
      if (r == 0)
        k_affine_round<F, true><<<lay.grid, AFF_THREADS, AffStage<F>::BYTES, s>>>(bases, entries, off0, off_out, c.k0, c.k1, out,
                                                                 r < R - 1, prefix);
      else
        k_affine_round<F, false><<<lay.grid, AFF_THREADS, AffStage<F>::BYTES, s>>>(buf[(r - 1) & 1], nullptr, off_out - (K + 1),
                                                                  off_out, c.k0, c.k1, out, r < R - 1, prefix);
    }
    *launches += R;
  }
  return cudaGetLastError();
}

}  // namespace gm
