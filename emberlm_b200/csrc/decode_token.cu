// Persistent token kernel of the preset decoders: batch-1 greedy generation, or one chosen token.
//
// A token is a chain of small dependent products (per layer: QKV rows, attention, O rows, gate|up rows,
// down rows), each a few microseconds of weight streaming spread over the whole chip, so what bounds it is
// the hand-over of the vector between two products. One CTA of 16 warps per SM owns the same contiguous
// rows of every matrix throughout, and vectors travel as words {value, number of the exchange}: a producer
// stores its rows with 64-bit relaxed stores, a consumer polls the words it needs until all carry the
// number it waits for. That is one trip through L2 per hand-over. The grid barrier that this replaces took
// three dependent ones (release and add, poll, load of the vector) and added up 296 arrivals on one
// address: 6.8 us a hand-over, 1.33 ms a token for Qwen3-0.6B (28 layers, 256 + 128 tokens) and 1.08 ms for
// SmolLM2-135M against 0.37 and 0.08 ms of weight streaming.
//
// While a CTA waits for a vector, the first weights of its rows are on their way into registers and the
// chunks of the product after the next are on their way into L2 (one bulk prefetch instruction per 32 KB).
// The residual rows of a CTA stay in its shared memory; the RMSNorm factor is applied to the finished dot
// products, so a vector is staged with one block barrier.
//
// Why a buffer can be overwritten without an acknowledgement: every CTA owns at least one row of each
// product (token_grid), so a complete vector implies that every CTA has finished the phase that read the
// vector before it; between two uses of one buffer there are at least two such complete vectors.
// Every wait is bounded (Patience).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdint>

#include "decode_token.h"

namespace ctdk {
namespace {

constexpr int kThreads = 512, kWarps = 16;
constexpr int kMaxUnits = 1024;        // (row, part) pairs of one CTA in one product
constexpr int kMaxRows = 512;          // residual rows of a CTA
constexpr int kPre = 8;                // 16-byte weight loads of a warp lane in flight
constexpr int kHeads = 4;              // query heads per pass over the keys
constexpr int kAbort = 2;

__device__ __forceinline__ void put(Word* w, float v, unsigned epoch) {
  const Word x = (static_cast<Word>(epoch) << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(x) : "memory");
}
__device__ __forceinline__ Word get(const Word* w) {
  Word x;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(w) : "memory");
  return x;
}
__device__ __forceinline__ void get2(const Word* w, Word& x, Word& y) {   // w 16-byte aligned; each word is whole, the pair need not be
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(w) : "memory");
}
__device__ __forceinline__ bool is_from(Word x, unsigned epoch) { return static_cast<unsigned>(x >> 32) == epoch; }
__device__ __forceinline__ float value_of(Word x) { return __uint_as_float(static_cast<unsigned>(x)); }

// The rare part of a wait, out of line: a token runs through far more code than the instruction caches hold close, and
// every wait has one. True when the thread gives up: another one has, or kMostPolls (some seconds) have been made
// since the last block barrier, which sets the status word and the abort flag that makes all CTAs leave.
constexpr unsigned kMostPolls = 1u << 23;
__device__ __noinline__ bool wait_is_over(unsigned int* sync, int* status, unsigned polls) {
  if (ld_acquire_u32(sync + kAbort) != 0u) return true;
  if (polls < kMostPolls) return false;
  if (atomicCAS(status, 0, CTDK_ETIMEOUT) == 0) {
    status[1] = 90;
    status[2] = static_cast<int>(blockIdx.x);
    status[3] = static_cast<int>(threadIdx.x);
  }
  atomicExch(sync + kAbort, 1u);
  return true;
}
// The bound of a thread's waits: more() says whether to poll on. Once it has said no it keeps to that; the
// block agrees on leaving at the next barrier (left()).
struct Patience {
  unsigned int* sync;
  int* status;
  bool gone = false;
  unsigned polls = 0;
  __device__ __forceinline__ Patience(const TokenKernelArgs& a) : sync(a.sync), status(a.status) {}
  __device__ __forceinline__ bool more() {
    if ((++polls & 63u) == 0u && wait_is_over(sync, status, polls)) gone = true;
    return !gone;
  }
  // Block barrier; true when any thread gave up. The count starts anew.
  __device__ __forceinline__ bool left() {
    polls = 0;
    return __syncthreads_or(gone) != 0;
  }
};

// f(i, value i, value i + 1) for the words w[0, n) (n even), dealt to the block in pairs with four pairs of a
// thread in flight, once they carry `epoch`.
template <class F>
__device__ __forceinline__ void take(const Word* w, int n, unsigned epoch, Patience& p, F f) {
  constexpr int U = 4, kStep = 2 * kThreads;
  for (int base = 2 * threadIdx.x; base < n; base += kStep * U) {
    Word x[U], y[U];
    unsigned open = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = y[u] = 0ull;
      if (base + kStep * u < n) open |= 1u << u;
    }
    while (true) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (open >> u & 1u) get2(w + base + kStep * u, x[u], y[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((open >> u & 1u) && is_from(x[u], epoch) && is_from(y[u], epoch)) {
          open &= ~(1u << u);
          f(base + kStep * u, value_of(x[u]), value_of(y[u]));
        }
      if (open == 0u || !p.more()) break;
    }
  }
}

// [first, first + count) of n items for this CTA; every CTA gets at least one when n >= gridDim.x.
struct Share {
  int first, count;
  __device__ __forceinline__ Share(int n) {
    first = static_cast<int>(static_cast<int64_t>(n) * blockIdx.x / gridDim.x);
    count = static_cast<int>(static_cast<int64_t>(n) * (blockIdx.x + 1) / gridDim.x) - first;
  }
};

// Requests [p, p + bytes) into L2, one instruction of up to 32 KB per lane; called by one warp. A CTA asks for
// at most 64 KB a call: up to five calls (QKV, O, gate, up, down) are outstanding, 47 MB over the grid of a 126 MB L2
// that keeps lines read from both halves twice. Qwen3-1.7B, 100 + 16 tokens: 28.7 ms with 256 KB a call, 27.1 with 128,
// 26.7 with 64; Qwen3-0.6B, 100 + 32: 27.9, 27.9, 27.7.
__device__ __forceinline__ void ask(const void* p, int64_t bytes) {
  const int lane = threadIdx.x & 31;
  constexpr int64_t kPiece = 32768, kMost = 65536;
  if (bytes > kMost) bytes = kMost;
  const int64_t at = lane * kPiece;
  if (at >= bytes) return;
  const unsigned n = static_cast<unsigned>(bytes - at < kPiece ? bytes - at : kPiece) & ~15u;
  if (n != 0u)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const char*>(p) + at), "r"(n) : "memory");
}
__device__ __forceinline__ void ask_rows(const float* W, const Share& r, int K) {
  ask(W + static_cast<int64_t>(r.first) * K, static_cast<int64_t>(r.count) * K * 4);
}

// The products y = W v of this CTA's rows: unit u = (virtual row u >> s, part u & (2^s - 1)) belongs to warp
// u mod 16; s_part[u] receives the unit's sum. Virtual rows are rows of w0, or with w1 alternately rows of
// w0 and w1. start() requests the first weights of the warp's first unit, before the vector is there.
struct Product {
  const float *w0, *w1;
  int K4, s, units;
  float4 pre[kPre];

  __device__ __forceinline__ Product(const float* a, const float* b, const Share& r, int K, int s_)
      : w0(a + static_cast<int64_t>(r.first) * K), w1(b == nullptr ? nullptr : b + static_cast<int64_t>(r.first) * K), K4(K / 4), s(s_),
        units((b == nullptr ? r.count : 2 * r.count) << s_) {}
  __device__ __forceinline__ const float4* row(int u) const {
    const int v = u >> s;
    const float* p = w1 == nullptr ? w0 + static_cast<int64_t>(v) * K4 * 4 : ((v & 1) ? w1 : w0) + static_cast<int64_t>(v >> 1) * K4 * 4;
    return reinterpret_cast<const float4*>(p);
  }
  __device__ __forceinline__ int lo(int u) const { return ((u & ((1 << s) - 1)) * K4) >> s; }
  __device__ __forceinline__ int hi(int u) const { return (((u & ((1 << s) - 1)) + 1) * K4) >> s; }
  __device__ __forceinline__ void load(int u) {
    const float4* p = row(u);
    const int end = hi(u), i0 = lo(u) + (threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < kPre; ++j) pre[j] = i0 + 32 * j < end ? __ldcs(p + i0 + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void start() {
    const int u = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < kPre; ++j) pre[j] = make_float4(0.f, 0.f, 0.f, 0.f);   // defined on every path: otherwise live from the kernel's start
    if (u < units) load(u);
  }
  __device__ __forceinline__ void finish(const float* xs, float* s_part) {
    const int lane = threadIdx.x & 31;
    const float4* x4 = reinterpret_cast<const float4*>(xs);
    for (int u = threadIdx.x >> 5; u < units; u += kWarps) {
      const float4* p = row(u);
      const int end = hi(u), i0 = lo(u) + lane;
      float acc = 0.0f, acc2 = 0.0f;
#pragma unroll
      for (int j = 0; j < kPre; ++j) {
        const int i = i0 + 32 * j;
        if (i < end) {
          const float4 v = x4[i], w = pre[j];
          acc = fmaf(w.x, v.x, acc);
          acc2 = fmaf(w.y, v.y, acc2);
          acc = fmaf(w.z, v.z, acc);
          acc2 = fmaf(w.w, v.w, acc2);
        }
        if (j & 1) asm volatile("" ::: "memory");   // at most two chunks of the vector in registers at a time
      }
      for (int i = i0 + 32 * kPre; i < end; i += 32 * kPre) {
        float4 w[kPre];
#pragma unroll
        for (int j = 0; j < kPre; ++j) w[j] = i + 32 * j < end ? __ldcs(p + i + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < kPre; ++j) {
          if (i + 32 * j < end) {
            const float4 v = x4[i + 32 * j];
            acc = fmaf(w[j].x, v.x, acc);
            acc2 = fmaf(w[j].y, v.y, acc2);
            acc = fmaf(w[j].z, v.z, acc);
            acc2 = fmaf(w[j].w, v.w, acc2);
          }
          if (j & 1) asm volatile("" ::: "memory");
        }
      }
      if (u + kWarps < units) load(u + kWarps);   // under the reduction of this unit
      acc = warp_sum(acc + acc2);
      if (lane == 0) s_part[u] = acc;
    }
  }
  // Sum of virtual row v's parts.
  __device__ __forceinline__ float sum(const float* s_part, int v) const {
    float t = 0.0f;
    for (int k = 0; k < (1 << s); ++k) t += s_part[(v << s) + k];
    return t;
  }
};

// DC consecutive floats of a head row per lane (head size 32 DC).
template <int DC>
struct Vec {
  float v[DC];
  __device__ __forceinline__ void load(const float* row, int lane) {
    if (DC == 2) {
      const float2 t = __ldcg(reinterpret_cast<const float2*>(row) + lane);
      v[0] = t.x;
      v[1] = t.y;
    } else {
      const float4 t = __ldcg(reinterpret_cast<const float4*>(row) + lane);
      v[0] = t.x;
      v[1] = t.y;
      v[2 % DC] = t.z;
      v[3 % DC] = t.w;
    }
  }
  __device__ __forceinline__ void shared(const float* row, int lane) {
#pragma unroll
    for (int c = 0; c < DC; ++c) v[c] = row[lane * DC + c];
  }
};

// Key ranges per kv head for L keys. One range needs no merge (a hand-over of ~1 us less); above 96 KB of
// keys and values (1 us of one SM's L2 bandwidth) the heads are cut into ranges of about 24 KB.
__device__ __forceinline__ int attn_splits(int L, int D, int Hk) {
  const int64_t bytes = static_cast<int64_t>(L) * D * 8;
  int most = gridDim.x / Hk;
  if (most > kTokenMaxSplits) most = kTokenMaxSplits;
  if (bytes <= 98304 || most < 2) return 1;
  const int want = static_cast<int>((bytes + 24575) / 24576);
  return want < most ? want : most;
}

struct Shared {
  float* xs;      // the staged vector, or the attention's scratch
  float* part;    // [kMaxUnits]
  float* res;     // [kMaxRows] residual rows of this CTA
  float* red;     // [kWarps]
};

// Heads of kv head hk against keys [j0, j1); results as words of the attention vector (whole) or of the range.
template <int DC>
__device__ __noinline__ bool attention_item(const TokenKernelArgs& a, int l, int hk, int sp, int splits, int pos, unsigned e_qkv, unsigned e_part,
                               unsigned e_attn, const Shared& sh, Patience& p) {
  constexpr int U = 4, D = 32 * DC;   // keys of a warp in flight; head size
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int G = a.H / a.Hk, L = pos + 1;
  const int per = (L + splits - 1) / splits;
  const int j0 = min(L, sp * per), j1 = min(L, j0 + per);
  const bool has_new = pos >= j0 && pos < j1;
  const TokenLayer& w = a.lw[l];
  float* qs = sh.xs;                     // [G][D]
  float* kn = qs + G * D;                // [D] new key
  float* vn = kn + D;                    // [D] new value
  float* scr = vn + D;                   // [16][kHeads][D + 2]
  const int64_t layer = (static_cast<int64_t>(l) * a.Hk + hk) * a.max_seq * D;
  float* kc = a.kcache + layer;
  float* vc = a.vcache + layer;
  const float2* cs_row = a.table + static_cast<int64_t>(pos) * (D / 2);

  // new rows: a warp per head; queries 0 .. G-1, then key and value where the range holds the new position
  for (int r = wid; r < G + (has_new ? 2 : 0); r += kWarps) {
    const int head = r < G ? hk * G + r : (r == G ? a.H + hk : a.H + a.Hk + hk);
    const Word* src = a.qkv + static_cast<int64_t>(head) * D;
    // angles and norm weights are requested before the wait
    float2 cs[DC / 2];
    float nw[DC], x[DC];
#pragma unroll
    for (int c = 0; c < DC / 2; ++c) cs[c] = __ldg(cs_row + lane + 32 * c);
#pragma unroll
    for (int c = 0; c < DC; ++c) {
      nw[c] = a.qk_norm && r <= G ? __ldg(a.P + (r < G ? w.wqn : w.wkn) + lane + 32 * c) : 1.0f;
      x[c] = 0.0f;
    }
    unsigned open = (1u << DC) - 1u;
    while (true) {
      Word word[DC] = {};
#pragma unroll
      for (int c = 0; c < DC; ++c)
        if (open >> c & 1u) word[c] = get(src + lane + 32 * c);
#pragma unroll
      for (int c = 0; c < DC; ++c)
        if ((open >> c & 1u) && is_from(word[c], e_qkv)) {
          x[c] = value_of(word[c]);
          open &= ~(1u << c);
        }
      if (open == 0u || !p.more()) break;
    }
    __syncwarp();
    float* dst = r < G ? qs + r * D : (r == G ? kn : vn);
    if (r <= G) {   // per-head RMSNorm, then rotation of the pairs (i, i + D / 2)
      if (a.qk_norm) {
        float ss = 0.0f;
#pragma unroll
        for (int c = 0; c < DC; ++c) ss += x[c] * x[c];
        const float s = rsqrtf(warp_sum(ss) / static_cast<float>(D) + a.eps);
#pragma unroll
        for (int c = 0; c < DC; ++c) x[c] = x[c] * s * nw[c];
      }
#pragma unroll
      for (int c = 0; c < DC / 2; ++c) {
        const float u = x[c], v = x[c + DC / 2];
        x[c] = u * cs[c].x - v * cs[c].y;
        x[c + DC / 2] = u * cs[c].y + v * cs[c].x;
      }
    }
#pragma unroll
    for (int c = 0; c < DC; ++c) dst[lane + 32 * c] = x[c];
    if (r >= G) {
      float* cache = (r == G ? kc : vc) + static_cast<int64_t>(pos) * D;
#pragma unroll
      for (int c = 0; c < DC; ++c) cache[lane + 32 * c] = x[c];
    }
  }
  if (p.left()) return false;

  const int stride = D + 2;
  for (int g0 = 0; g0 < G; g0 += kHeads) {
    float q[kHeads][DC], m[kHeads], s[kHeads], o[kHeads][DC];
#pragma unroll
    for (int g = 0; g < kHeads; ++g) {
      m[g] = -FLT_MAX;
      s[g] = 0.0f;
#pragma unroll
      for (int c = 0; c < DC; ++c) {
        q[g][c] = g0 + g < G ? qs[(g0 + g) * D + lane * DC + c] * a.scale : 0.0f;
        o[g][c] = 0.0f;
      }
    }
    for (int jb = j0 + wid; jb < j1; jb += kWarps * U) {
      Vec<DC> k[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = jb + kWarps * u;
        if (j < j1 && j != pos) {
          k[u].load(kc + static_cast<int64_t>(j) * D, lane);
          v[u].load(vc + static_cast<int64_t>(j) * D, lane);
        } else {
          k[u].shared(kn, lane);
          v[u].shared(vn, lane);
        }
      }
      float d[U][kHeads];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int g = 0; g < kHeads; ++g) {
          float t = 0.0f;
#pragma unroll
          for (int c = 0; c < DC; ++c) t = fmaf(q[g][c], k[u].v[c], t);
          d[u][g] = g0 + g < G ? warp_sum(t) : 0.0f;
        }
#pragma unroll
      for (int g = 0; g < kHeads; ++g) {
        if (g0 + g >= G) continue;
        float mx = m[g];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (jb + kWarps * u < j1) mx = fmaxf(mx, d[u][g]);
        const float fix = __expf(m[g] - mx);
        s[g] *= fix;
#pragma unroll
        for (int c = 0; c < DC; ++c) o[g][c] *= fix;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (jb + kWarps * u < j1) {
            const float e = __expf(d[u][g] - mx);
            s[g] += e;
#pragma unroll
            for (int c = 0; c < DC; ++c) o[g][c] = fmaf(e, v[u].v[c], o[g][c]);
          }
        m[g] = mx;
      }
    }
#pragma unroll
    for (int g = 0; g < kHeads; ++g) {
      if (g0 + g >= G) continue;
      float* dst = scr + (wid * kHeads + g) * stride;
      if (lane == 0) {
        dst[0] = m[g];
        dst[1] = s[g];
      }
#pragma unroll
      for (int c = 0; c < DC; ++c)
        dst[2 + lane * DC + c] = o[g][c];
    }
    __syncthreads();
    const int heads = G - g0 < kHeads ? G - g0 : kHeads;
    for (int i = threadIdx.x; i < heads * D; i += kThreads) {
      const int g = i / D, e = i - g * D, h = hk * G + g0 + g;
      const float* src = scr + g * stride;
      float M = -FLT_MAX;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) M = fmaxf(M, src[k * kHeads * stride]);
      float sum = 0.0f, out = 0.0f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) {
        const float f = __expf(src[k * kHeads * stride] - M);
        sum = fmaf(f, src[k * kHeads * stride + 1], sum);
        out = fmaf(f, src[k * kHeads * stride + 2 + e], out);
      }
      if (splits == 1) {
        put(a.attn + static_cast<int64_t>(h) * D + e, out / sum, e_attn);
      } else {
        Word* dst = a.part + (static_cast<int64_t>(h) * kTokenMaxSplits + sp) * stride;
        put(dst + 2 + e, out, e_part);
        if (e == 0) {
          put(dst, j0 < j1 ? M : -FLT_MAX, e_part);
          put(dst + 1, j0 < j1 ? sum : 0.0f, e_part);
        }
      }
    }
    __syncthreads();   // scr, and before another item the staged rows, are written again
  }
  return true;
}

// Merges the ranges of 32 columns of one head (a warp).
__device__ __forceinline__ void merge_columns(const TokenKernelArgs& a, int h, int col, int splits, unsigned e_part, unsigned e_attn, Patience& p) {
  const int lane = threadIdx.x & 31, stride = a.D + 2;
  const Word* src = a.part + static_cast<int64_t>(h) * kTokenMaxSplits * stride;
  float m = -FLT_MAX, l = 0.0f;
  if (lane < splits) {
    while (true) {
      const Word x = get(src + lane * stride), y = get(src + lane * stride + 1);
      if (is_from(x, e_part) && is_from(y, e_part)) {
        m = value_of(x);
        l = value_of(y);
        break;
      }
      if (!p.more()) break;
    }
  }
  __syncwarp();
  const float M = warp_max(m);
  const float f = lane < splits ? __expf(m - M) : 0.0f;
  const float inv = 1.0f / warp_sum(f * l);
  const int c = col + lane;
  float out = 0.0f;
  constexpr int U = 8;
  for (int s0 = 0; s0 < splits; s0 += U) {
    float v[U];
    unsigned open = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      v[u] = 0.0f;
      if (s0 + u < splits) open |= 1u << u;
    }
    while (open != 0u) {
      Word x[U] = {};
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (open >> u & 1u) x[u] = get(src + static_cast<int64_t>(s0 + u) * stride + 2 + c);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((open >> u & 1u) && is_from(x[u], e_part)) {
          v[u] = value_of(x[u]);
          open &= ~(1u << u);
        }
      if (open != 0u && !p.more()) break;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float fu = __shfl_sync(0xffffffffu, f, (s0 + u) & 31);
      if (s0 + u < splits) out = fmaf(fu, v[u], out);
    }
  }
  put(a.attn + static_cast<int64_t>(h) * a.D + c, out * inv, e_attn);
}

template <int DC>
__global__ void __launch_bounds__(kThreads, 1) token_kernel(const __grid_constant__ TokenKernelArgs a) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_part[kMaxUnits];
  __shared__ float s_res[kMaxRows];
  __shared__ float s_red[kWarps];
  __shared__ Word s_best[kWarps];
  const Shared sh{sm, s_part, s_res, s_red};
  Patience p(a);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int D = 32 * DC;
  const int hid = a.hid, I = a.I, HD = a.H * D;
  const Share r_qkv(a.QKVN), r_hid(hid), r_i(I), r_v(a.V);
  int pos = a.counters[0];
  int64_t tok = *a.cur_token;
  unsigned e = 0;   // number of the last exchange
  if (wid == 0) {
    ask_rows(a.P + a.lw[0].wq, r_qkv, hid);
    ask_rows(a.P + a.lw[0].wo, r_hid, HD);
  }

  // xs = v * nw for the words of an exchange, or for plain values (null: zeros); s_red collects the sum of squares of
  // v. False: the block leaves.
  auto stage_norm = [&](const Word* words, const float* plain, unsigned epoch, const float* nw) {
    float ss = 0.0f;
    auto store = [&](int i, float u, float v) {
      const float2 n = __ldg(reinterpret_cast<const float2*>(nw + i));
      *reinterpret_cast<float2*>(sm + i) = make_float2(u * n.x, v * n.y);
      ss = fmaf(u, u, fmaf(v, v, ss));
    };
    if (words != nullptr) take(words, hid, epoch, p, store);
    else
      for (int i = 2 * threadIdx.x; i < hid; i += 2 * kThreads)
        store(i, plain != nullptr ? __ldg(plain + i) : 0.0f, plain != nullptr ? __ldg(plain + i + 1) : 0.0f);
    ss = warp_sum(ss);
    if (lane == 0) s_red[wid] = ss;
    return !p.left();
  };
  auto norm_factor = [&]() {
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) t += s_red[k];
    return rsqrtf(t / static_cast<float>(hid) + a.eps);
  };
  auto stage = [&](const Word* words, int n, unsigned epoch) {
    take(words, n, epoch, p, [&](int i, float u, float v) { *reinterpret_cast<float2*>(sm + i) = make_float2(u, v); });
    return !p.left();
  };

  for (int t = 0; t < a.n_tokens; ++t) {
    // layer 0 reads the embedding row in place; a given id outside the vocabulary is a row of zeros and is counted, as
    // in embedding_fwd_kernel
    const bool known = tok >= 0 && tok < a.V;
    const float* row = known ? a.P + a.embed + tok * hid : nullptr;
    if (!known && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.status[2], 1);
    for (int i = threadIdx.x; i < r_hid.count; i += kThreads) s_res[i] = known ? row[r_hid.first + i] : 0.0f;
    const int L = pos + 1, splits = attn_splits(L, D, a.Hk), items = a.Hk * splits;
    for (int l = 0; l < a.L; ++l) {
      const TokenLayer& w = a.lw[l];
      const unsigned e_x = e, e_qkv = e + 1, e_part = e + 2, e_attn = e + 3, e_hm = e + 4, e_act = e + 5;
      e += 6;   // the last one: the residual stream behind this layer
      // ---- qkv = Wqkv rmsnorm(x) ----
      {
        Product pr(a.P + w.wq, nullptr, r_qkv, hid, a.s_qkv);
        pr.start();
        if (wid == kWarps - 1) {
          ask_rows(a.P + w.wg, r_i, hid);
          ask_rows(a.P + w.wg + static_cast<int64_t>(I) * hid, r_i, hid);
        }
        if (!stage_norm(l > 0 ? a.x : nullptr, row, e_x, a.P + w.w_in)) return;
        pr.finish(sm, s_part);
        __syncthreads();
        const float sc = norm_factor();
        for (int r = threadIdx.x; r < r_qkv.count; r += kThreads) put(a.qkv + r_qkv.first + r, pr.sum(s_part, r) * sc, e_qkv);
      }
      // ---- attention of the new row ----
      for (int item = blockIdx.x; item < items; item += gridDim.x) {
        if (!attention_item<DC>(a, l, item / splits, item % splits, splits, pos, e_qkv, e_part, e_attn, sh, p)) return;
      }
      Product p_o(a.P + w.wo, nullptr, r_hid, HD, a.s_o);
      p_o.start();
      if (wid == kWarps - 1) ask_rows(a.P + w.wd, r_hid, I);
      if (splits > 1) {
        // a warp per 32 columns of a head, spread from the last CTA on (the first ones have the items)
        const int cols = DC, from_end = gridDim.x - 1 - blockIdx.x;
        for (int u = from_end + wid * gridDim.x; u < a.H * cols; u += gridDim.x * kWarps)
          merge_columns(a, u / cols, (u % cols) * 32, splits, e_part, e_attn, p);
      }
      // ---- hm = x + Wo attn ----
      if (!stage(a.attn, HD, e_attn)) return;
      p_o.finish(sm, s_part);
      __syncthreads();
      for (int r = threadIdx.x; r < r_hid.count; r += kThreads) {
        const float v = s_res[r] + p_o.sum(s_part, r);
        s_res[r] = v;
        put(a.hm + r_hid.first + r, v, e_hm);
      }
      // ---- act = silu(gate) * up of Wgu rmsnorm(hm) ----
      {
        Product pr(a.P + w.wg, a.P + w.wg + static_cast<int64_t>(I) * hid, r_i, hid, a.s_gu);
        pr.start();
        if (wid == kWarps - 1) {
          if (l + 1 < a.L) {
            ask_rows(a.P + a.lw[l + 1].wq, r_qkv, hid);
            if (static_cast<int>(blockIdx.x) < items) {
              const int hk = blockIdx.x / splits, sp = blockIdx.x % splits, per = (L + splits - 1) / splits;
              const int j0 = min(L, sp * per), j1 = min(L, j0 + per);
              const int64_t at = ((static_cast<int64_t>(l + 1) * a.Hk + hk) * a.max_seq + j0) * D;
              ask(a.kcache + at, static_cast<int64_t>(j1 - j0) * D * 4);
              ask(a.vcache + at, static_cast<int64_t>(j1 - j0) * D * 4);
            }
            if (blockIdx.x == gridDim.x - 1) {
              ask(a.P + a.lw[l + 1].w_in, hid * 4);
              ask(a.P + a.lw[l + 1].w_post, hid * 4);
            }
          } else {
            ask_rows(a.P + a.embed, r_v, hid);
          }
        }
        if (!stage_norm(a.hm, nullptr, e_hm, a.P + w.w_post)) return;
        pr.finish(sm, s_part);
        __syncthreads();
        const float sc = norm_factor();
        for (int r = threadIdx.x; r < r_i.count; r += kThreads) {
          const float g = pr.sum(s_part, 2 * r) * sc, u = pr.sum(s_part, 2 * r + 1) * sc;
          put(a.act + r_i.first + r, g / (1.0f + __expf(-g)) * u, e_act);
        }
      }
      // ---- x = hm + Wd act ----
      {
        Product pr(a.P + w.wd, nullptr, r_hid, I, a.s_d);
        pr.start();
        if (wid == kWarps - 1 && l + 1 < a.L) ask_rows(a.P + a.lw[l + 1].wo, r_hid, HD);
        if (!stage(a.act, I, e_act)) return;
        pr.finish(sm, s_part);
        __syncthreads();
        for (int r = threadIdx.x; r < r_hid.count; r += kThreads) {
          const float v = s_res[r] + pr.sum(s_part, r);
          s_res[r] = v;
          put(a.x + r_hid.first + r, v, e);
        }
      }
    }

    // ---- tied LM head and arg-max (first index of the maximum): a warp per pair of rows ----
    if (!stage_norm(a.x, nullptr, e, a.P + a.norm)) return;
    const float sc = norm_factor();
    Word best = 0ull;
    {
      const float* E = a.P + a.embed + static_cast<int64_t>(r_v.first) * hid;
      const float4* x4 = reinterpret_cast<const float4*>(sm);
      const int K4 = hid / 4;
      for (int n = 2 * wid; n < r_v.count; n += 2 * kWarps) {
        const float4* p0 = reinterpret_cast<const float4*>(E + static_cast<int64_t>(n) * hid);
        const bool two = n + 1 < r_v.count;
        const float4* p1 = two ? p0 + K4 : p0;
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 8
        for (int i = lane; i < K4; i += 32) {
          const float4 u = __ldcs(p0 + i), v = __ldcs(p1 + i), x = x4[i];
          a0 = fmaf(u.x, x.x, fmaf(u.y, x.y, fmaf(u.z, x.z, fmaf(u.w, x.w, a0))));
          a1 = fmaf(v.x, x.x, fmaf(v.y, x.y, fmaf(v.z, x.z, fmaf(v.w, x.w, a1))));
        }
        a0 = warp_sum(a0) * sc;
        a1 = warp_sum(a1) * sc;
        if (lane == 0) {
          const int at = r_v.first + n;
          a.logits[at] = a0;
          Word k = argmax_key(a0, at);
          best = k > best ? k : best;
          if (two) {
            a.logits[at + 1] = a1;
            k = argmax_key(a1, at + 1);
            best = k > best ? k : best;
          }
        }
      }
    }
    if (a.out_tokens == nullptr) return;
    if (lane == 0) s_best[wid] = best;
    if (wid == kWarps - 1 && t + 1 < a.n_tokens) {
      ask_rows(a.P + a.lw[0].wq, r_qkv, hid);
      ask_rows(a.P + a.lw[0].wo, r_hid, HD);
    }
    __syncthreads();
    const unsigned e_best = ++e;
    if (threadIdx.x == 0) {
#pragma unroll
      for (int k = 1; k < kWarps; ++k) best = s_best[k] > best ? s_best[k] : best;
      // this CTA's new cache rows, written in front of block barriers, are read by other CTAs from the next token on:
      // the fence stands in the thread that publishes
      __threadfence();
      put(a.best + 2 * blockIdx.x, __uint_as_float(static_cast<unsigned>(best >> 32)), e_best);
      put(a.best + 2 * blockIdx.x + 1, __uint_as_float(static_cast<unsigned>(best)), e_best);
    }
    best = 0ull;
    take(a.best, 2 * static_cast<int>(gridDim.x), e_best, p, [&](int, float h, float lo) {
      const Word k = (static_cast<Word>(__float_as_uint(h)) << 32) | __float_as_uint(lo);
      best = k > best ? k : best;
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const Word k = __shfl_xor_sync(0xffffffffu, best, o);
      best = k > best ? k : best;
    }
    if (p.left()) return;   // and thread 0 has read s_best
    if (lane == 0) s_best[wid] = best;
    __threadfence();   // behind the words of all CTAs: their new cache rows are visible from here on
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kWarps; ++k) best = s_best[k] > best ? s_best[k] : best;
    tok = static_cast<int64_t>(0xFFFFFFFFu - static_cast<unsigned>(best & 0xFFFFFFFFull));
    if (blockIdx.x == 0 && threadIdx.x == 0) a.out_tokens[a.out_offset + t] = tok;
    pos += 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.counters[0] = pos;
    a.counters[1] += a.n_tokens;
    *a.cur_token = tok;
  }
}

using Kernel = void (*)(TokenKernelArgs);
Kernel kernel_of(int D) {
  return D == 64 ? token_kernel<2> : token_kernel<4>;
}
size_t shared_bytes(const TokenKernelArgs& a) {
  const int64_t stage = std::max(std::max(a.hid, a.H * a.D), a.I);
  const int64_t attn = static_cast<int64_t>(a.H / a.Hk + 2) * a.D + static_cast<int64_t>(kWarps) * kHeads * (a.D + 2);
  return static_cast<size_t>(std::max(stage, attn)) * sizeof(float);
}
// Warps per row: the split whose longest warp reads least (whole rounds of 16 warps), the smaller one on a tie, among
// those whose parts are one batch of loads (kPre, 1024 values): a further batch is only requested when the one before has
// been multiplied, so its whole latency is exposed. Qwen3-1.7B (rows of 2048 and 6144), 100 + 16 tokens: 41.5 ms without
// that condition, 27.1 with it; with batches of 512, 32.2. Parts stay longer where kMaxUnits allows no finer split.
int row_split(int rows, int K) {
  int best = 0;
  int64_t least = INT64_MAX;
  for (int s = 0; s <= 4; ++s) {
    const int64_t rounds = ((static_cast<int64_t>(rows) << s) + kWarps - 1) / kWarps;
    // a round also costs a reduction and a staggered start, about as long as two loads
    const int64_t cost = rounds * ((K / 4 + (32 << s) - 1) / (32 << s) + 2);
    const bool last = s == 4 || (static_cast<int64_t>(rows) << (s + 1)) > kMaxUnits;
    if (cost < least && (last || (K / 4 + (1 << s) - 1) >> s <= 32 * kPre) && (static_cast<int64_t>(rows) << s) <= kMaxUnits) {
      least = cost;
      best = s;
    }
  }
  return best;
}
int64_t padded(int64_t n) { return (n + 31) / 32 * 32; }

}  // namespace

int64_t token_words(int hid, int QKVN, int I, int H, int D) {
  return 2 * padded(hid) + padded(QKVN) + padded(static_cast<int64_t>(H) * kTokenMaxSplits * (D + 2)) + padded(static_cast<int64_t>(H) * D) +
         padded(I) + padded(2 * kTokenMaxGrid);
}

static void token_carve(TokenKernelArgs& a, Word* words) {
  a.x = words;
  a.hm = a.x + padded(a.hid);
  a.qkv = a.hm + padded(a.hid);
  a.part = a.qkv + padded(a.QKVN);
  a.attn = a.part + padded(static_cast<int64_t>(a.H) * kTokenMaxSplits * (a.D + 2));
  a.act = a.attn + padded(static_cast<int64_t>(a.H) * a.D);
  a.best = a.act + padded(a.I);
}

int token_grid(const TokenKernelArgs& a) {
  const int D = a.D;
  const bool shape = a.L <= kTokenMaxLayers && a.hid % 8 == 0 && (a.H * D) % 8 == 0 && a.I % 8 == 0 && (D == 64 || D == 128) && a.H <= 96;
  int dev = 0, coop = 0, per_sm = 0;
  const size_t smem = shared_bytes(a);
  if (!shape || smem > 160 * 1024) return 0;
  const void* k = reinterpret_cast<const void*>(kernel_of(D));
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || coop == 0 ||
      raise_dynamic_smem(k, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  // every CTA owns at least one row of each product (the protocol needs that)
  const int grid = std::min(std::min(std::min(sm_count(), kTokenMaxGrid), a.hid), std::min(std::min(a.I, a.QKVN), a.V));
  const int rows = std::max(std::max(ceil_div(a.QKVN, grid), 2 * ceil_div(a.I, grid)), ceil_div(a.hid, grid));
  return rows <= kMaxUnits && ceil_div(a.hid, grid) <= kMaxRows ? grid : 0;
}

int token_launch(TokenKernelArgs& a, Word* words, int grid, cudaStream_t s) {
  a.s_qkv = row_split(ceil_div(a.QKVN, grid), a.hid);
  a.s_o = row_split(ceil_div(a.hid, grid), a.H * a.D);
  a.s_gu = row_split(2 * ceil_div(a.I, grid), a.hid);
  a.s_d = row_split(ceil_div(a.hid, grid), a.I);
  token_carve(a, words);
  a.status = device_status_word();
  if (a.status == nullptr) return fail(CTDK_ELAUNCH, "decode: no status word");
  // exchanges are numbered from 1 in every launch: no word of an earlier one may carry a number
  const int64_t bytes = token_words(a.hid, a.QKVN, a.I, a.H, a.D) * static_cast<int64_t>(sizeof(Word));
  if (cudaMemsetAsync(words, 0, bytes, s) != cudaSuccess || cudaMemsetAsync(a.sync, 0, 16 * sizeof(unsigned int), s) != cudaSuccess)
    return fail(CTDK_ELAUNCH, "decode: clearing the exchange words failed");
  void* params[] = {&a};
  const cudaError_t err = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel_of(a.D)), dim3(grid), dim3(kThreads), params,
                                                      shared_bytes(a), s);
  if (err != cudaSuccess) return fail(CTDK_ELAUNCH, "decode: cooperative launch failed: %s", cudaGetErrorString(err));
  return check_launch("decode token kernel");
}

}  // namespace ctdk
