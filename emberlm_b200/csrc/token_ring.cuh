// The weight ring of the persistent token kernels (decode_token.cu, hybrid_token.cu).
//
// A token is a chain of small products, each a few microseconds of weight streaming over the whole chip behind a
// hand-over of the vector. Weights do not depend on the vector, so one warp per CTA requests the CTA's rows of every
// product, in the order of the phases, with bulk copies into a ring of stages in shared memory, as far ahead as the ring
// reaches (100 to 180 KB per SM, 15 to 27 MB over the chip: one or two phases), while the compute warps wait for vectors.
// What a phase then still takes is one pass over shared memory. Every wait is bounded.
#pragma once

#include <algorithm>
#include <climits>
#include <cstdint>

#include <cuda_bf16.h>

#include "decode_core.h"

namespace ctdk {

// Compute warps; one more requests weights. Eight, not sixteen: what a warp does per phase beside its loads is the same for
// few and for many of them, and sixteen and one leave 96 registers a thread, so that the kernels spilled into an L1 of which
// the ring leaves 28 KB.
constexpr int kRingWarps = 8, kRingThreads = 32 * kRingWarps;
constexpr int kRingMaxStages = 16;
constexpr int kRingAbort = 2;         // word of the abort flag among the sync words

// A product's rows in the ring: a row of `chunks` 16-byte chunks belongs to one warp (row v of a CTA to warp v mod 8) and
// passes in `pieces` pieces; a stage holds one piece of eight rows. Whole rows, although four of eight warps may have none in
// a small product: parts of a row on several warps would need a block barrier and another trip through shared memory before
// a result can leave.
struct RingRows {
  int chunks, pieces, len;   // len: chunks of a piece, the last one has what is left
};
inline RingRows ring_rows(int chunks, int piece) {
  const int pieces = ceil_div(chunks, piece), len = ceil_div(chunks, pieces);
  return RingRows{chunks, ceil_div(chunks, len), len};
}
inline int ring_stage_bytes(const RingRows& r) { return kRingWarps * r.len * 16; }

#ifdef __CUDACC__

// Barriers of the compute warps (W of them). The instructions want whole warps: lanes that a poll or a store of one lane has
// split off come back first.
template <int W = kRingWarps>
__device__ __forceinline__ void ring_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory");
}
template <int W = kRingWarps>
__device__ __forceinline__ bool ring_or(bool x) {
  unsigned r;
  __syncwarp();
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
               : "=r"(r)
               : "r"(static_cast<unsigned>(x)), "n"(32 * W)
               : "memory");
  return r != 0u;
}

// Barrier words: [0] arrivals, [kRingAbort] abort flag (all zero at launch).
// The compute warps of all CTAs of a cooperative grid meet here: one release reduction on a counter per CTA (no value
// comes back, so the arriving thread does not wait for it; the CTA's earlier writes are ordered
// before it by the bar.sync and the release), then one thread per CTA polls the counter. A flag per
// CTA watched by every other CTA measured twice as slow (all pollers hit the same few L2 lines).
// Arrival and wait are two calls, with whatever does not depend on the others between them. `epoch` counts the barriers this
// CTA has passed. Bounded: when the wait runs out, the status word gets `where` and the abort flag makes every CTA leave at
// its next barrier. The wait returns false once any CTA has given up: the caller unwinds.
template <int W = kRingWarps>
__device__ __forceinline__ void grid_arrive(unsigned int* sync, unsigned int& epoch) {
  ring_sync<W>();
  ++epoch;
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&sync[0]) : "memory");
}
static __device__ __noinline__ bool grid_wait_longer(unsigned int* sync, int* status, int where, unsigned int target) {
  const uint64_t t0 = globaltimer_ns();
  unsigned int spins = 0;
  while (ld_acquire_u32(&sync[0]) < target) {
    if ((++spins & 0xffu) != 0u) continue;
    if (ld_acquire_u32(&sync[kRingAbort]) != 0u) return false;   // someone else gave up
    if (globaltimer_ns() - t0 > kWaitBudgetNs) {
      if (atomicCAS(status, 0, CTDK_ETIMEOUT) == 0) {
        status[1] = where;
        status[2] = static_cast<int>(blockIdx.x);
      }
      atomicExch(&sync[kRingAbort], 1u);
      return false;
    }
  }
  return true;
}
template <int W = kRingWarps>
__device__ __forceinline__ bool grid_wait(unsigned int* sync, int* status, int where, unsigned int epoch) {
  bool gone = false;
  if (threadIdx.x == 0) {
    const unsigned int target = epoch * gridDim.x;
    bool there = false;
#pragma unroll 1
    for (int i = 0; i < 64 && !there; ++i) there = ld_acquire_u32(&sync[0]) >= target;
    gone = (!there && !grid_wait_longer(sync, status, where, target)) || ld_acquire_u32(&sync[kRingAbort]) != 0u;
  }
  return !ring_or<W>(gone);
}

// Waits on the ring: the rare part is out of line.
static __device__ __noinline__ bool ring_wait_longer(uint64_t* bar, uint32_t parity, unsigned int* sync, int* status) {
  const uint64_t t0 = globaltimer_ns();
  unsigned int spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((spins++ & 63u) != 0u) continue;
    if (ld_acquire_u32(&sync[kRingAbort]) != 0u) return false;   // someone gave up
    if (globaltimer_ns() - t0 > kWaitBudgetNs) {
      if (atomicCAS(status, 0, CTDK_ETIMEOUT) == 0) {
        status[1] = 90;
        status[2] = static_cast<int>(blockIdx.x);
        status[3] = static_cast<int>(threadIdx.x);
      }
      atomicExch(&sync[kRingAbort], 1u);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, unsigned int* sync, int* status) {
  return mbar_try_wait(bar, parity) || ring_wait_longer(bar, parity, sync, status);
}

// A stage is full when its copies have landed and free when every compute warp has read it. Each side keeps its own place.
struct Ring {
  char* at;
  uint64_t *full, *free;   // [stages]
  int stages, bytes;
  unsigned int* sync;
  int* status;
  int stage = 0;
  unsigned parity = 0;
  __device__ __forceinline__ Ring(char* at_, uint64_t* bars /* [2 kRingMaxStages] */, int stages_, int bytes_, unsigned int* sync_, int* status_)
      : at(at_), full(bars), free(bars + kRingMaxStages), stages(stages_), bytes(bytes_), sync(sync_), status(status_) {}
  __device__ __forceinline__ void init() {   // one thread; the block meets before the ring is used
    for (int i = 0; i < stages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(free + i, kRingWarps);
    }
    mbar_fence_init();
  }
  __device__ __forceinline__ void next() {
    if (++stage == stages) {
      stage = 0;
      parity ^= 1u;
    }
  }
  __device__ __forceinline__ char* here() const { return at + static_cast<int64_t>(stage) * bytes; }
};

// The weights are read once a token: they leave the L2 first, which keeps vectors, caches and states there.
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// The requesting warp's side.
struct RingRequests {
  Ring ring;
  uint64_t policy;
  int pending = 0;   // stages requested so far, up to the ring's length
  __device__ __forceinline__ explicit RingRequests(const Ring& r) : ring(r), policy(evict_first_policy()) {}
  // `rows` rows from row `first` of w0; with w1, eight of w0 and the same eight of w1 in turn. False when a wait ran out.
  __device__ __forceinline__ bool rows(const char* w0, const char* w1, int64_t first, int rows, const RingRows& r) {
    const int lane = threadIdx.x & 31;
    w0 += first * r.chunks * 16;
    if (w1 != nullptr) w1 += first * r.chunks * 16;
#pragma unroll 1
    for (int v0 = 0; v0 < rows; v0 += kRingWarps) {
      const int n = min(kRingWarps, rows - v0);
#pragma unroll 1
      for (const char* w = w0; w != nullptr; w = w == w0 ? w1 : nullptr) {
#pragma unroll 1
        for (int piece = 0; piece < r.pieces; ++piece) {
          if (!__all_sync(0xffffffffu, ring_wait(ring.free + ring.stage, ring.parity ^ 1u, ring.sync, ring.status))) return false;
          const int lo = piece * r.len, len = min(r.len, r.chunks - lo);
          uint64_t* bar = ring.full + ring.stage;
          if (lane == 0) mbar_expect_tx(bar, static_cast<unsigned>(n * len) * 16u);
          __syncwarp();
          const char* src = w + (static_cast<int64_t>(v0) * r.chunks + lo) * 16;
          if (r.pieces == 1) {   // the rows lie side by side
            if (lane == 0) bulk_load(ring.here(), src, static_cast<unsigned>(n * len) * 16u, bar, policy);
          } else if (lane < n) {
            bulk_load(ring.here() + lane * len * 16, src + static_cast<int64_t>(lane) * r.chunks * 16, static_cast<unsigned>(len) * 16u, bar, policy);
          }
          ring.next();
          pending = min(pending + 1, ring.stages);
        }
      }
    }
    return true;
  }
  // A wait ran out: copies in flight land before the CTA ends.
  __device__ __forceinline__ void give_up() {
    for (; pending > 0; --pending) {
      if (--ring.stage < 0) {
        ring.stage = ring.stages - 1;
        ring.parity ^= 1u;
      }
      mbar_wait_bounded_w(ring.full + ring.stage, ring.parity, ring.status, 90);
    }
  }
};

// A 16-byte chunk of weights against the vector's values.
template <typename T>
struct RingChunk;
template <>
struct RingChunk<float> {
  static constexpr int kN = 4;
  __device__ __forceinline__ static void dot(const uint4& w, const float (&x)[4], float (&s)[4]) {
    ffma2(s[0], s[1], __uint_as_float(w.x), __uint_as_float(w.y), x[0], x[1], s[0], s[1]);
    ffma2(s[2], s[3], __uint_as_float(w.z), __uint_as_float(w.w), x[2], x[3], s[2], s[3]);
  }
};
template <>
struct RingChunk<__nv_bfloat16> {
  static constexpr int kN = 8;
  __device__ __forceinline__ static void dot(const uint4& w, const float (&x)[8], float (&s)[4]) {
    auto two = [](uint32_t u, float a, float b, float& s0, float& s1) {
      ffma2(s0, s1, __uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u), a, b, s0, s1);
    };
    two(w.x, x[0], x[1], s[0], s[1]);
    two(w.y, x[2], x[3], s[2], s[3]);
    two(w.z, x[4], x[5], s[0], s[1]);
    two(w.w, x[6], x[7], s[2], s[3]);
  }
};

// This CTA's rows of a product with the staged vector: f(row, sum, 0), or with a pair of matrices f(row, sum of the first,
// sum of the second), by one lane for each row. C: 16-byte chunks of a lane in a piece. The sums over the lanes of four turns
// share shuffles (seven instead of twenty), and each sum stands in a lane of its own, so that what f does with it is done once
// for four turns: against two turns at a time with eight lanes for a row, zutalix-0.6b 300 + 64 tokens 69.3 -> 65.0 ms,
// Qwen3-0.6B 256 + 128 89.5 -> 88.6, SmolLM2-360M single steps 14.75 -> 14.3. False when a wait ran out.
template <typename T, int C, class F>
__device__ __forceinline__ bool ring_multiply(Ring& ring, const RingRows& r, int rows, bool pairs, const float* xs, F f) {
  constexpr int N = RingChunk<T>::kN;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int turns = ((rows + kRingWarps - 1) / kRingWarps) << (pairs ? 1 : 0);
  float x[C][N];
  bool ok = true;
  int n = 0, len = 0;   // this lane's chunks of the piece: 0, 32, ... below n
  auto values = [&](int piece) {
    const int lo = piece * r.len;
    len = min(r.len, r.chunks - lo);
    n = len - lane;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int e = 0; e < N; e += 4) {
        const float4 v = 32 * c < n ? *reinterpret_cast<const float4*>(xs + (lo + lane + 32 * c) * N + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[c][e] = v.x;
        x[c][e + 1] = v.y;
        x[c][e + 2] = v.z;
        x[c][e + 3] = v.w;
      }
  };
  // a warp without a row multiplies what the stage holds in its place, which goes nowhere
  auto stage = [&](float (&s)[4]) {
    ok = ring_wait(ring.full + ring.stage, ring.parity, ring.sync, ring.status) && ok;
    const uint4* w4 = reinterpret_cast<const uint4*>(ring.here()) + wid * len + lane;
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (32 * c < n) RingChunk<T>::dot(w4[32 * c], x[c], s);
    __syncwarp();
    if (lane == 0) mbar_arrive(ring.free + ring.stage);
    ring.next();
  };
  values(0);
#pragma unroll 1
  for (int turn = 0; turn < turns; turn += 4) {
    float a[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      a[b] = 0.0f;
      if (turn + b >= turns) continue;
      float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (r.pieces == 1) {
        stage(s);
      } else {
#pragma unroll 1
        for (int piece = 0; piece < r.pieces; ++piece) {
          values(piece);
          stage(s);
        }
      }
      a[b] = (s[0] + s[2]) + (s[1] + s[3]);
    }
    // lanes 0 .. 7 have the sum of a[0], 16 .. 23 of a[1], 8 .. 15 of a[2], 24 .. 31 of a[3]
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    const float v0 = (h16 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, h16 ? a[0] : a[1], 16);
    const float v1 = (h16 ? a[3] : a[2]) + __shfl_xor_sync(0xffffffffu, h16 ? a[2] : a[3], 16);
    float v = (h8 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, h8 ? v0 : v1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const float behind = __shfl_xor_sync(0xffffffffu, v, 16);
    const int of = turn + (lane >> 4) + ((lane >> 2) & 2), row = (pairs ? of >> 1 : of) * kRingWarps + wid;
    if ((lane & 7) == 0 && row < rows && of < turns && !(pairs && lane >= 16)) f(row, v, behind);
  }
  return ok;
}

#endif

}  // namespace ctdk
