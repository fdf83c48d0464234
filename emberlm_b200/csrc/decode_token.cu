// Persistent token kernel of the preset decoders: batch-1 greedy generation, or one chosen token.
//
// A token is a chain of small dependent products (per layer: QKV rows, attention, O rows, gate|up rows, down rows), each a
// few microseconds of weight streaming spread over the whole chip, so what bounds it is the hand-over of the vector between
// two products. One CTA per SM owns the same contiguous rows of every matrix throughout, and vectors travel as words
// {value, number of the exchange}: a producer puts its rows with 64-bit reductions, a consumer polls the words it needs until
// all carry the number it waits for. That is one trip through L2 per hand-over, about 2000 cycles for 1024 words.
//
// The weights stream through shared memory meanwhile (token_ring.cuh): when a vector is there, a phase is one pass over them.
// A phase is executed once per layer by two warps of a scheduler, a dependent chain of instructions at five to eight cycles
// each, so the instructions of the chain are what the rest of a phase costs: one body for all products, a row per warp whose
// sum leaves without another barrier, a RMSNorm factor that is applied to the finished sums, no integer divisions (200
// cycles each) and nothing in local memory (the ring leaves 28 KB of L1).
// Qwen3-0.6B, 256 + 128 tokens: 109.3 -> 90.2 ms against sixteen warps with the weights in registers and plain stores of the
// words; SmolLM2-135M, 37 + 48: 26.2 -> 20.4; SmolLM2-360M, 700 + 16 single steps: 17.6 -> 14.0.
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
#include "mma_bf16.cuh"

namespace ctdk {
namespace {

constexpr int kThreads = kRingThreads, kWarps = kRingWarps;   // that compute; one more warp requests weights
constexpr int kLaneChunks = 8;         // 16-byte chunks of a lane in a piece: 32 values of the vector in registers

// A later exchange has the larger number, so the maximum replaces the word. Not a store: the rows of two CTAs share 32-byte
// sectors, and stores of parts of a sector from different SMs hold each other up. One exchange over 148 CTAs with nothing
// else, cycles with stores and with reductions: 576 words (whole sectors) 1800 and 1930, 1024 words 3780 and 2050, 2048
// words 3520 and 2500, 3072 words 4020 and 3020; a counter barrier and loads 3270 to 3800.
__device__ __forceinline__ void put(Word* w, float v, unsigned epoch) {
  const Word x = (static_cast<Word>(epoch) << 32) | __float_as_uint(v);
  asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(w), "l"(x) : "memory");
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
  if (ld_acquire_u32(sync + kRingAbort) != 0u) return true;
  if (polls < kMostPolls) return false;
  if (atomicCAS(status, 0, CTDK_ETIMEOUT) == 0) {
    status[1] = 90;
    status[2] = static_cast<int>(blockIdx.x);
    status[3] = static_cast<int>(threadIdx.x);
  }
  atomicExch(sync + kRingAbort, 1u);
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
    return ring_or(gone);
  }
};

__device__ __forceinline__ void get4(const Word* w, Word (&x)[4]) {   // w 32-byte aligned; each word is whole
  asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3]) : "l"(w) : "memory");
}

// f(i, the four values from i on, their weights) for the words w[0, n) (n a multiple of four, w 32-byte aligned), dealt to the
// block in fours with U of a thread in flight, once they carry `epoch`. The weights nw (null: ones) are requested before the
// wait.
template <class F>
__device__ __forceinline__ void take(const Word* w, const float* nw, int n, unsigned epoch, Patience& p, F f) {
  constexpr int U = 2, kStep = 4 * kThreads;
#pragma unroll 1
  for (int base = 4 * threadIdx.x; base < n; base += kStep * U) {
    Word x[U][4];
    float4 factor[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      factor[u] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      if (nw != nullptr && base + kStep * u < n) factor[u] = __ldg(reinterpret_cast<const float4*>(nw + base + kStep * u));
    }
    bool all;
    do {
      all = true;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (base + kStep * u < n) get4(w + base + kStep * u, x[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (base + kStep * u < n) all = all && is_from(x[u][0], epoch) && is_from(x[u][1], epoch) && is_from(x[u][2], epoch) && is_from(x[u][3], epoch);
    } while (!all && p.more());
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (base + kStep * u < n) f(base + kStep * u, make_float4(value_of(x[u][0]), value_of(x[u][1]), value_of(x[u][2]), value_of(x[u][3])), factor[u]);
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

// Requests [p, p + bytes) into L2, one instruction of up to 32 KB per lane; called by one warp.
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

// The requesting warp (token_ring.cuh): this CTA's rows of all phases, for all tokens.
__device__ __forceinline__ void request_weights(const TokenKernelArgs& a, const Ring& ring) {
  RingRequests q(ring);
  const Share r_qkv(a.QKVN), r_hid(a.hid), r_i(a.I), r_v(a.V);
  for (int t = 0; t < a.n_tokens; ++t)
    for (int step = 0; step <= 4 * a.L; ++step) {
      const int j = step == 4 * a.L ? 4 : step & 3;
      const TokenLayer& w = a.lw[min(step >> 2, a.L - 1)];
      const Share& r = j == 0 ? r_qkv : (j == 2 ? r_i : (j == 4 ? r_v : r_hid));
      const float* w0 = a.P + (j == 0 ? w.wq : (j == 1 ? w.wo : (j == 2 ? w.wg : (j == 3 ? w.wd : a.embed))));
      const float* w1 = j == 2 ? w0 + static_cast<int64_t>(a.I) * a.hid : nullptr;
      if (!q.rows(reinterpret_cast<const char*>(w0), reinterpret_cast<const char*>(w1), r.first, r.count, a.product[j])) {
        q.give_up();
        return;
      }
    }
}

// Keys and values of TILE bytes stand in shared memory at a time, in two places: one tile is on its way while the other is read.
__device__ __forceinline__ constexpr int tile_keys(int D, int TILE) { return TILE / (8 * D); }

// Key ranges per kv head for L keys: of about kRangeKeys, as far as there are CTAs. A range more costs little, a merge is one
// hand-over, and the scores and sums of 16 keys take a CTA about 1000 cycles: SmolLM2-135M with 37 to 85 keys on one CTA per
// kv head took 13 200 cycles a layer.
constexpr int kRangeKeys = 16;
__device__ __forceinline__ int attn_splits(int L, int parts) {   // called once a token; parts: of all query heads
  int most = gridDim.x / parts;
  if (most > kTokenMaxSplits) most = kTokenMaxSplits;
  if (L <= kRangeKeys || most < 2) return 1;
  return min(most, (L + kRangeKeys - 1) / kRangeKeys);
}

// An item: query heads [head, head + heads) of kv head hk against keys [j0, j1), range sp; the first ones of a kv head write its new
// row. Made once a token: a phase has no time for the divisions (about 200 cycles each).
struct Item {
  int hk, head, heads, sp, j0, j1;
  bool writes;
  __device__ __forceinline__ Item(const TokenKernelArgs& a, int item, int splits, int L) {
    const int per = (L + splits - 1) / splits, of = item / splits;
    hk = of / a.head_groups;
    const int part = of - hk * a.head_groups, first = a.group * part / a.head_groups;
    head = hk * a.group + first;
    heads = a.group * (part + 1) / a.head_groups - first;
    writes = part == 0;
    sp = item - of * splits;
    j0 = min(L, sp * per);
    j1 = min(L, j0 + per);
  }
};

// Tile number n of an item, into its place ([tile_keys][D] keys, then values): always one group of copies, empty behind the
// last tile. The row of the new position comes from the QKV product.
template <int D, int TILE>
__device__ __forceinline__ void request_tile(const TokenKernelArgs& a, float* tiles, int l, const Item& it, int pos, int n) {
  constexpr int kKeys = tile_keys(D, TILE);
  const int j = it.j0 + n * kKeys, floats = min(kKeys, min(it.j1, pos) - j) * D;
  const int64_t at = ((static_cast<int64_t>(l) * a.Hk + it.hk) * a.max_seq + j) * D;
  const float *k = a.kcache + at, *v = a.vcache + at;
  float* tile = tiles + (n & 1) * (TILE / 4);
#pragma unroll 2
  for (int i = 4 * threadIdx.x; i < floats; i += 4 * kThreads) {
    cp_async16(tile + i, k + i);
    cp_async16(tile + TILE / 8 + i, v + i);
  }
  cp_async_commit();
}

inline __host__ __device__ int attention_scratch(int blocks) { return (blocks > kWarps ? blocks : kWarps) * 34; }

// Scores of n keys of a tile with all query heads, sc[head][key]: 16 threads per key, four sums of NH heads and 4 / NH keys at a
// time, whose reductions share shuffles (five in a chain of four instead of sixteen in a row). With that, eight keys' products in
// flight and one walk over the keys for all heads of a group, us a token behind 4000, 8000 and 16 000 positions: four layers of
// Llama-3-8B's sizes 690 -> 644, Qwen3-0.6B 1475 -> 1265, Llama-3.2-1B 1984 -> 1651.
template <int DC, int NH, int KEYS>
__device__ __forceinline__ void tile_scores(const float* tile, const float* qs, float* sc, int G, int n) {
  constexpr int D = 32 * DC, NK = 4 / NH;
  const int t = threadIdx.x & 15;
  const bool h8 = (t & 8) != 0, h4 = (t & 4) != 0;
  const int which = (h4 ? 2 : 0) + (h8 ? 1 : 0), my_key = kThreads / 16 * (which / NH), my_head = which % NH;   // of this thread's sum
#pragma unroll 1
  for (int key = threadIdx.x >> 4; (key & ~1) < n; key += kThreads / 16 * NK) {   // whole warps
    float4 k[NK][DC / 2];
#pragma unroll
    for (int x = 0; x < NK; ++x) {
      const int at = key + kThreads / 16 * x;
      const float4* k4 = reinterpret_cast<const float4*>(tile + (at < n ? at : 0) * D) + t;
#pragma unroll
      for (int c = 0; c < DC / 2; ++c) k[x][c] = k4[16 * c];
    }
#pragma unroll 1
    for (int g = 0; g < G; g += NH) {
      float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        const float4* q4 = reinterpret_cast<const float4*>(qs + min(g + h, G - 1) * D) + t;
#pragma unroll
        for (int c = 0; c < DC / 2; ++c) {
          const float4 q = q4[16 * c];
#pragma unroll
          for (int x = 0; x < NK; ++x)
            d[x * NH + h] = fmaf(q.x, k[x][c].x, fmaf(q.y, k[x][c].y, fmaf(q.z, k[x][c].z, fmaf(q.w, k[x][c].w, d[x * NH + h]))));
        }
      }
      const float d0 = (h8 ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, h8 ? d[0] : d[1], 8);
      const float d1 = (h8 ? d[3] : d[2]) + __shfl_xor_sync(0xffffffffu, h8 ? d[2] : d[3], 8);
      float v = (h4 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, h4 ? d0 : d1, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      if ((t & 3) == 0 && key + my_key < n && g + my_head < G) sc[(g + my_head) * KEYS + key + my_key] = v;
    }
  }
}

// Attention of the new row for one item, whose first two tiles have been requested: results as words of the attention vector
// (one range) or of the range. Threads: 16 per key for the scores; for the weighted sums a warp per 32 columns of a head
// and share of the keys.
template <int DC, int TILE>
__device__ __noinline__ bool attention_item(const TokenKernelArgs& a, int l, const Item it, int splits, int pos, unsigned e, int64_t wqn, int64_t wkn,
                                            float* sm, float* tiles) {
  constexpr int D = 32 * DC, kKeys = tile_keys(D, TILE);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, G = it.heads;
  Patience p(a);
  const bool has_new = pos >= it.j0 && pos < it.j1;
  float* qs = sm;                  // [G][D] rotated, scaled
  float* sc = qs + G * D;          // [G][kKeys] scores
  float* scr = sc + G * kKeys;     // [kWarps or blocks][34] partial results of the shares of the keys, or of the blocks
  float* kn = scr + attention_scratch(G * DC);   // [2][D] the new row
  // new rows: a warp per head; queries 0 .. G-1, then key and value where the range holds the new position
#pragma unroll 1
  for (int r = wid; r < G + (has_new ? 2 : 0); r += kWarps) {
    const int head = r < G ? it.head + r : (r == G ? a.H + it.hk : a.H + a.Hk + it.hk);
    const Word* src = a.qkv + static_cast<int64_t>(head) * D + lane;
    // angles and norm weights are requested before the wait
    float2 cs[DC / 2];
    float nw[DC], x[DC];
    const float* norm = a.P + (r < G ? wqn : wkn) + lane;
    const bool normed = a.qk_norm && r <= G;
#pragma unroll
    for (int c = 0; c < DC / 2; ++c) cs[c] = __ldg(a.table + static_cast<int64_t>(pos) * (D / 2) + lane + 32 * c);
#pragma unroll
    for (int c = 0; c < DC; ++c) nw[c] = normed ? __ldg(norm + 32 * c) : 1.0f;
    Word word[DC];
    bool all;
    do {
      all = true;
#pragma unroll
      for (int c = 0; c < DC; ++c) word[c] = get(src + 32 * c);
#pragma unroll
      for (int c = 0; c < DC; ++c) all = all && is_from(word[c], e + 1);
    } while (!all && p.more());
    __syncwarp();
    float ss = 0.0f;
#pragma unroll
    for (int c = 0; c < DC; ++c) {
      x[c] = value_of(word[c]);
      ss += x[c] * x[c];
    }
    if (r <= G) {   // per-head RMSNorm, then rotation of the pairs (i, i + D / 2)
      if (normed) {
        const float s = rsqrtf(warp_sum(ss) * (1.0f / D) + a.eps);
#pragma unroll
        for (int c = 0; c < DC; ++c) x[c] = x[c] * s * nw[c];
      }
      const float f = r < G ? a.scale : 1.0f;
#pragma unroll
      for (int c = 0; c < DC / 2; ++c) {
        const float u = x[c], v = x[c + DC / 2];
        x[c] = (u * cs[c].x - v * cs[c].y) * f;
        x[c + DC / 2] = (u * cs[c].y + v * cs[c].x) * f;
      }
    }
    float* dst = (r < G ? qs + r * D : kn + (r - G) * D) + lane;
#pragma unroll
    for (int c = 0; c < DC; ++c) dst[32 * c] = x[c];
    if (r >= G && it.writes) {
      float* cache = (r == G ? a.kcache : a.vcache) + ((static_cast<int64_t>(l) * a.Hk + it.hk) * a.max_seq + pos) * D + lane;
#pragma unroll
      for (int c = 0; c < DC; ++c) cache[32 * c] = x[c];
    }
  }
  if (p.left()) return false;

  // blocks of 32 columns of a head, a warp each, with shares of the keys (the largest power of two that the warps allow); where
  // there are more blocks than warps, a warp takes several, whose sums stand in its places of `scr` between two tiles
  const int blocks = G * DC, turns = (blocks + kWarps - 1) / kWarps;
  const int sh = blocks * 8 <= kWarps ? 3 : (blocks * 4 <= kWarps ? 2 : (blocks * 2 <= kWarps ? 1 : 0)), shares = 1 << sh;
  int mine_first = wid, share = 0;   // this warp's first block
  if (turns == 1) {
#pragma unroll 1
    for (; mine_first >= blocks; mine_first -= blocks) ++share;
  }
  float m = -FLT_MAX, s = 0.0f, o = 0.0f;
#pragma unroll 1
  for (int j = it.j0, number = 0; j < it.j1; j += kKeys, ++number) {
    const int n = min(kKeys, it.j1 - j);
    float* const tile = tiles + (number & 1) * (TILE / 4);
    cp_async_wait<1>();
    ring_sync();
    if (pos >= j && pos < j + n) {
      if (threadIdx.x < 2 * D) tile[(threadIdx.x < D ? 0 : TILE / 8) + (pos - j) * D + (threadIdx.x & (D - 1))] = kn[threadIdx.x];
      ring_sync();
    }
    if (G == 1) tile_scores<DC, 1, kKeys>(tile, qs, sc, 1, n);
    else if (G == 2) tile_scores<DC, 2, kKeys>(tile, qs, sc, 2, n);
    else tile_scores<DC, 4, kKeys>(tile, qs, sc, G, n);
    ring_sync();
    if (share < shares) {
      const int mine = (n - share + shares - 1) >> sh;   // keys share, share + shares, ... of the tile
#pragma unroll 1
      for (int blk = mine_first; blk < blocks; blk += kWarps) {
        const int h = blk / DC, col = blk % DC * 32 + lane;
        float* const held = scr + blk * 34;
        if (turns > 1 && j != it.j0) {
          m = held[0];
          s = held[1];
          o = held[2 + lane];
        }
#pragma unroll 1
        for (int i0 = 0; i0 < mine; i0 += 32) {
          const int count = min(32, mine - i0), first = share + i0 * shares;
          const float d = lane < count ? sc[h * kKeys + first + lane * shares] : -FLT_MAX;
          const float most = fmaxf(m, warp_max(d)), w = lane < count ? __expf(d - most) : 0.0f, fix = __expf(m - most);
          m = most;
          s = s * fix + warp_sum(w);
          o *= fix;
          const float* v = tile + TILE / 8 + first * D + col;
#pragma unroll 8
          for (int i = 0; i < count; ++i) o = fmaf(__shfl_sync(0xffffffffu, w, i), v[i * shares * D], o);
        }
        if (turns > 1) {
          __syncwarp();   // all lanes have read the maximum and the sum
          held[2 + lane] = o;
          if (lane == 0) *reinterpret_cast<float2*>(held) = make_float2(m, s);
          __syncwarp();
          m = -FLT_MAX;
          s = o = 0.0f;
        }
      }
    }
    const bool more = j + 2 * kKeys < it.j1;
    if (more) ring_sync();   // this place has been read
    request_tile<D, TILE>(a, tiles, l, it, more ? pos : 0, number + 2);
  }
  if (shares > 1) {
    scr[wid * 34 + 2 + lane] = o;
    if (lane == 0) *reinterpret_cast<float2*>(scr + wid * 34) = make_float2(m, s);
    ring_sync();
    if (share == 0) {
#pragma unroll 1
      for (int k = 1; k < shares; ++k) {
        const float* other = scr + (wid + k * blocks) * 34;
        const float most = fmaxf(m, other[0]), f = __expf(m - most), fo = __expf(other[0] - most);
        s = s * f + other[1] * fo;
        o = o * f + other[2 + lane] * fo;
        m = most;
      }
    }
  }
  if (share == 0) {
#pragma unroll 1
    for (int blk = mine_first; blk < blocks; blk += kWarps) {
      const int head = it.head + blk / DC, col = blk % DC * 32 + lane;
      if (turns > 1 && it.j0 < it.j1) {
        const float* held = scr + blk * 34;
        m = held[0];
        s = held[1];
        o = held[2 + lane];
      }
      if (splits == 1) {
        put(a.attn + head * D + col, o / s, e + 3);
      } else {   // [column][range]: the ranges of a column side by side
        Word* dst = a.part + (static_cast<int64_t>(head) * (D + 2)) * kTokenMaxSplits + it.sp;
        put(dst + col * kTokenMaxSplits, o, e + 2);
        if (col == 0) {
          put(dst + D * kTokenMaxSplits, it.j0 < it.j1 ? m : -FLT_MAX, e + 2);
          put(dst + (D + 1) * kTokenMaxSplits, s, e + 2);
        }
      }
    }
  }
  ring_sync();   // the scratch is written again
  return !p.gone;
}

// Merges the ranges of a column of a head: a lane per range.
__device__ __forceinline__ void merge_column(const TokenKernelArgs& a, int h, int col, int splits, unsigned e, Patience& p) {
  const int lane = threadIdx.x & 31;
  const Word* src = a.part + static_cast<int64_t>(h) * (a.D + 2) * kTokenMaxSplits + (lane < splits ? lane : 0);
  Word m, s, o;
  do {
    m = get(src + a.D * kTokenMaxSplits);
    s = get(src + (a.D + 1) * kTokenMaxSplits);
    o = get(src + col * kTokenMaxSplits);
  } while (!(is_from(m, e + 2) && is_from(s, e + 2) && is_from(o, e + 2)) && p.more());
  __syncwarp();
  const float most = warp_max(value_of(m)), f = lane < splits ? __expf(value_of(m) - most) : 0.0f;
  const float sum = warp_sum(f * value_of(s)), out = warp_sum(f * value_of(o));
  if (lane == 0) put(a.attn + h * a.D + col, out / sum, e + 3);
}

// What the compute warps look up per kind of phase (QKV, O, gate|up, down, head), in shared memory.
struct PhaseRows {
  RingRows rows;
  int first, count;   // of this CTA
};

template <int DC, int TILE>
__global__ void __launch_bounds__(kThreads + 32, 1) token_kernel(const __grid_constant__ TokenKernelArgs a) {
  // two places for the vector, under them the attention's scratch and tiles (plan), this CTA's residual rows, the ring
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(16) float s_red[kWarps];
  __shared__ Word s_best[kWarps];
  __shared__ uint64_t s_bar[2 * kRingMaxStages];
  __shared__ PhaseRows s_rows[5];
  __shared__ TokenLayer s_layer[kTokenMaxLayers];
  constexpr int D = 32 * DC;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, hid = a.hid;
  float *const tile = sm + a.tile_at, *const res = sm + a.front_floats;
  Ring ring(reinterpret_cast<char*>(res + a.residual_floats), s_bar, a.stages, a.stage_bytes, a.sync, a.status);
  if (threadIdx.x == 0) ring.init();
  if (threadIdx.x < 5) {
    const int j = threadIdx.x;
    const Share r(j == 0 ? a.QKVN : (j == 2 ? a.I : (j == 4 ? a.V : hid)));
    s_rows[j] = PhaseRows{a.product[j], r.first, r.count};
  }
  for (int l = threadIdx.x; l < a.L; l += kThreads + 32) s_layer[l] = a.lw[l];
  __syncthreads();
  if (wid == kWarps) {
    request_weights(a, ring);
    return;
  }
  Patience p(a);
  int pos = a.counters[0];
  int64_t tok = *a.cur_token;
  unsigned e = 0;   // number of the last exchange
  const float inv_hid = 1.0f / static_cast<float>(hid);

  // False: a wait ran out, here or in another CTA.
  auto tokens = [&]() {
#pragma unroll 1
    for (int t = 0; t < a.n_tokens; ++t) {
      // layer 0 reads the embedding row in place; a given id outside the vocabulary is a row of zeros and is counted, as
      // in embedding_fwd_kernel
      const bool known = tok >= 0 && tok < a.V;
      const float* row = known ? a.P + a.embed + tok * hid : nullptr;
      if (!known && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.status[2], 1);
      for (int i = threadIdx.x; i < s_rows[1].count; i += kThreads) res[i] = known ? row[s_rows[1].first + i] : 0.0f;
      const int parts = a.Hk * a.head_groups, splits = attn_splits(pos + 1, parts), items = parts * splits;
      const Item mine(a, blockIdx.x, splits, pos + 1);
      Word best = 0ull;
      // Exchanges of layer l: e + 1 qkv, e + 2 ranges, e + 3 attention, e + 4 hm, e + 5 act, e + 6 x. One body for all
      // products keeps the code that a token runs through small.
#pragma unroll 1
      for (int step = 0; step <= 4 * a.L; ++step) {
        const int j = step == 4 * a.L ? 4 : step & 3, l = min(step >> 2, a.L - 1);   // QKV, O, gate|up, down; the head
        if (j == 0 && static_cast<int>(blockIdx.x) < items) {   // cached rows, under the QKV product
          if (a.tiles_over != 0) ring_sync();   // the second place of the vector has been read
          request_tile<D, TILE>(a, tile, l, mine, pos, 0);
          request_tile<D, TILE>(a, tile, l, mine, pos, 1);
        }
        if (j == 1) {   // attention of the new row
#pragma unroll 1
          for (int item = blockIdx.x; item < items; item += gridDim.x) {
            ring_sync();   // the scratch lies over both places of the vector
            Item it = mine;
            if (item >= static_cast<int>(gridDim.x)) {
              it = Item(a, item, splits, pos + 1);
              request_tile<D, TILE>(a, tile, l, it, pos, 0);
              request_tile<D, TILE>(a, tile, l, it, pos, 1);
            }
            if (!attention_item<DC, TILE>(a, l, it, splits, pos, e, s_layer[l].wqn, s_layer[l].wkn, sm, tile)) return false;
          }
          if (splits > 1) {
            // columns are dealt from the last CTA on (the first ones have the items)
#pragma unroll 1
            for (int u = gridDim.x - 1 - blockIdx.x + wid * gridDim.x; u < a.H * D; u += gridDim.x * kWarps) merge_column(a, u / D, u % D, splits, e, p);
          }
        }
        if (j == 2 && blockIdx.x == gridDim.x - 1 && wid == kWarps - 1 && l + 1 < a.L) {   // norm weights, on their way into L2
          ask(a.P + s_layer[l + 1].w_in, hid * 4);
          ask(a.P + s_layer[l + 1].w_post, hid * 4);
        }
        // ---- the vector, in one of two places in turn: the other one may still be read. xs = v (times the norm weights; s_red collects the sum of squares of v) ----
        const bool normed = j != 1 && j != 3;
        float* const xs = sm + (normed ? 0 : a.second_at);
        {
          const float* nw = a.P + (j == 0 ? s_layer[l].w_in : (j == 2 ? s_layer[l].w_post : a.norm));
          float ss = 0.0f;
          auto store = [&](int i, float4 v, float4 f) {
            *reinterpret_cast<float4*>(xs + i) = make_float4(v.x * f.x, v.y * f.y, v.z * f.z, v.w * f.w);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
          };
          if (step > 0) {
            take((j == 1 ? a.attn : (j == 2 ? a.hm : (j == 3 ? a.act : a.x))), normed ? nw : nullptr, j == 1 ? a.H * D : (j == 3 ? a.I : hid),
                 normed && j != 2 ? e : e + (j == 1 ? 3u : (j == 2 ? 4u : 5u)), p, store);
          } else {
#pragma unroll 1
            for (int i = 4 * threadIdx.x; i < hid; i += 4 * kThreads)
              store(i, row != nullptr ? __ldg(reinterpret_cast<const float4*>(row + i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f),
                    __ldg(reinterpret_cast<const float4*>(nw + i)));
          }
          if (normed) {
            ss = warp_sum(ss);
            if (lane == 0) s_red[wid] = ss;
          }
          if (p.left()) return false;
        }
        float sc = 1.0f;   // the norm's factor, applied to the finished products
        if (normed) {
          const float4* r4 = reinterpret_cast<const float4*>(s_red);
          const float4 r0 = r4[0], r1 = r4[1];
          sc = rsqrtf((((r0.x + r0.y) + (r0.z + r0.w)) + ((r1.x + r1.y) + (r1.z + r1.w))) * inv_hid + a.eps);
        }
        const int first = s_rows[j].first;
        const bool glu = j == 2, added = j == 1 || j == 3;
        Word* const out = (j == 0 ? a.qkv : (j == 1 ? a.hm : (j == 2 ? a.act : a.x))) + first;
        const unsigned number = e + (j == 0 ? 1u : 3u + j);
        const bool ok = ring_multiply<float, kLaneChunks>(ring, s_rows[j].rows, s_rows[j].count, glu, xs, [&](int row, float v, float u) {
          v *= sc;
          if (j == 4) {   // tied LM head and arg-max (first index of the maximum)
            a.logits[first + row] = v;
            const Word k = argmax_key(v, first + row);
            best = k > best ? k : best;
            return;
          }
          // act = silu(gate) * up; the approximate division gives zero for divisors from 2^126 on, for 0.4 % of a token of SmolLM2-135M
          if (glu) v = v / (1.0f + __expf(-v)) * (u * sc);
          if (added) {   // the same lane has a row of O and of the down product
            v += res[row];
            res[row] = v;
          }
          put(out + row, v, number);
        });
        if (!ok) p.gone = true;
        if (a.second_at == 0) ring_sync();   // one place only: the vector has been read
        if (j == 3) e += 6;
      }
      if (a.out_tokens == nullptr) return true;
      // ---- the arg-max of all CTAs ----
      const unsigned e_best = ++e;
#pragma unroll 1
      for (int round = 0; round < 2; ++round) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const Word k = __shfl_xor_sync(0xffffffffu, best, o);
          best = k > best ? k : best;
        }
        if (lane == 0) s_best[wid] = best;
        // before round 0's words this CTA's new cache rows, written in front of block barriers, are read by other CTAs: the
        // fence stands in the thread that publishes; behind round 1's words those of all CTAs are visible from here on
        if (round == 1) __threadfence();
        if (p.left()) return false;
        best = s_best[lane & (kWarps - 1)];
#pragma unroll
        for (int o = kWarps / 2; o > 0; o >>= 1) {
          const Word k = __shfl_xor_sync(0xffffffffu, best, o);
          best = k > best ? k : best;
        }
        if (round == 1) break;
        if (threadIdx.x == 0) {
          __threadfence();
          Word* w = a.best + 2 * blockIdx.x;
          put(w, __uint_as_float(static_cast<unsigned>(best >> 32)), e_best);
          put(w + 1, __uint_as_float(static_cast<unsigned>(best)), e_best);
        }
        best = 0ull;
#pragma unroll 1
        for (int i = threadIdx.x; i < static_cast<int>(gridDim.x); i += kThreads) {
          Word x, y;
          do {
            get2(a.best + 2 * i, x, y);
          } while (!(is_from(x, e_best) && is_from(y, e_best)) && p.more());
          const Word k = (x << 32) | (y & 0xffffffffull);
          best = k > best ? k : best;
        }
        ring_sync();   // s_best has been read
      }
      tok = static_cast<int64_t>(0xFFFFFFFFu - static_cast<unsigned>(best & 0xFFFFFFFFull));
      if (blockIdx.x == 0 && threadIdx.x == 0) a.out_tokens[a.out_offset + t] = tok;
      pos += 1;
    }
    return true;
  };
  const bool done = tokens();
  cp_async_wait_all();   // a CTA that leaves early may have copies in flight
  if (!done) return;
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.out_tokens != nullptr) {
    a.counters[0] = pos;
    a.counters[1] += a.n_tokens;
    *a.cur_token = tok;
  }
}

using Kernel = void (*)(TokenKernelArgs);
constexpr int kTileBytes[2] = {32768, 16384};   // of a place
Kernel kernel_of(int D, int tile) {
  if (tile == kTileBytes[0]) return D == 64 ? token_kernel<2, kTileBytes[0]> : token_kernel<4, kTileBytes[0]>;
  return D == 64 ? token_kernel<2, kTileBytes[1]> : token_kernel<4, kTileBytes[1]>;
}
// Lays the shared memory out and returns its size (0: no room). The vectors of width hid stand in the first place and the
// other two, attention and act, in the second one, so that the places of a phase and the next differ; with one place a phase
// waits until the one before has read it. The attention's scratch lies over both places, its tiles behind them or (`over`, a
// block barrier more) over the second one: they are asked for while the QKV product reads the first, and have been read when the
// attention vector comes. The ring gets what is left, in pieces of up to `piece` chunks.
size_t lay_out(TokenKernelArgs& a, int grid, int tile, int places, bool over, int piece) {
  constexpr int64_t kRoom = 227 * 1024 - 4096;   // the kernel's own arrays take 3.1 KB
  auto up = [](int64_t n) { return (n + 31) / 32 * 32; };
  // With one or two key/value heads the ranges leave most CTAs without an item: their query heads are dealt to several. Four layers
  // behind 3000 positions, us a token: 32 heads of 128 on one key/value head (width 4096) 893 -> 674, 96 on one (2048) 1207 -> 418.
  a.group = a.H / a.Hk;
  a.head_groups = std::min(a.group, std::max(1, grid / (a.Hk * kTokenMaxSplits)));
  const int64_t first = up(a.hid), second = up(std::max(a.H * a.D, a.I)), G = ceil_div(a.group, a.head_groups);
  const int64_t scratch = up(G * (a.D + tile / (8 * a.D)) + attention_scratch(static_cast<int>(G) * a.D / 32) + 2 * a.D);
  a.tile_bytes = tile;
  a.residual_floats = static_cast<int>(up(ceil_div(a.hid, grid)));
  a.second_at = places == 2 ? static_cast<int>(first) : 0;
  const int64_t vectors = std::max(first, a.second_at + second), tiles = int64_t{2} * tile / 4;
  a.tile_at = static_cast<int>(std::max(over ? first : vectors, scratch));
  a.tiles_over = a.tile_at < vectors ? 1 : 0;
  a.front_floats = static_cast<int>(std::max(vectors, a.tile_at + tiles));
  const int64_t front = (a.front_floats + a.residual_floats) * int64_t{4};
  const int K[5] = {a.hid, a.H * a.D, a.hid, a.I, a.hid};
  a.stage_bytes = 0;
  for (int j = 0; j < 5; ++j) {
    a.product[j] = ring_rows(K[j] / 4, piece);
    a.stage_bytes = std::max(a.stage_bytes, ring_stage_bytes(a.product[j]));
  }
  a.stages = static_cast<int>(std::min<int64_t>((kRoom - front) / a.stage_bytes, kRingMaxStages));
  return a.stages >= 3 ? static_cast<size_t>(front + static_cast<int64_t>(a.stages) * a.stage_bytes) : 0;
}
// The longest pieces of which three stages fit, in two places rather than one, four stages rather than three, tiles of 32 KB where
// that leaves four stages, and of their own rather than over the second place. A stage costs the warps about the same whatever it
// holds, and what is on its way has to cover the memory's latency: four layers of Llama-3-8B's sizes (4096, 14336) took 833 us a
// token with four stages of 16 KB behind two places for any vector and tiles of their own, and take 567 with four of 32 KB; two
// layers of 8192 and 28672 1436 with four of 16 KB, 1007 with three of 32 KB and one place. Rows of 32768 leave five of 16 KB (four
// layers of width 1024: 437 us, 751 with eleven of 8 KB). Tiles of 32 KB over the second place against tiles of 16 KB beside it, us a
// token: Qwen3-1.7B behind 10, 300 and 4000 positions 1275, 1304, 1667 and 1272, 1335, 1833; Llama-3.2-1B behind 16 000 1651 and 1765.
size_t plan(TokenKernelArgs& a, int grid) {
  for (int piece = 32 * kLaneChunks; piece >= 32; piece /= 2)
    for (int places = 2; places >= 1; --places)
      for (int stages = 4; stages >= 3; --stages)
        for (int tile : kTileBytes)
          for (int over = 0; over <= 1; ++over) {
            const size_t size = lay_out(a, grid, tile, places, over != 0, piece);
            if (size != 0 && a.stages >= (tile == kTileBytes[0] ? 4 : stages)) return size;
          }
  return 0;
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

int token_grid(const TokenKernelArgs& args) {
  TokenKernelArgs a = args;
  const int D = a.D;
  const bool shape = a.L <= kTokenMaxLayers && a.hid % 8 == 0 && (a.H * D) % 8 == 0 && a.I % 8 == 0 && (D == 64 || D == 128) && a.H <= 96;
  int dev = 0, coop = 0, per_sm = 0;
  if (!shape) return 0;
  // every CTA owns at least one row of each product (the protocol needs that)
  const int grid = std::min(std::min(std::min(sm_count(), kTokenMaxGrid), a.hid), std::min(std::min(a.I, a.QKVN), a.V));
  const size_t smem = plan(a, grid);
  const void* k = reinterpret_cast<const void*>(kernel_of(D, a.tile_bytes));
  if (smem == 0 || cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      coop == 0 || raise_dynamic_smem(k, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads + 32, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  return grid;
}

int token_launch(TokenKernelArgs& a, Word* words, int grid, cudaStream_t s) {
  const size_t smem = plan(a, grid);
  CTDK_REQUIRE(smem != 0, "decode: no room for the weight ring");
  token_carve(a, words);
  a.status = device_status_word();
  if (a.status == nullptr) return fail(CTDK_ELAUNCH, "decode: no status word");
  // exchanges are numbered from 1 in every launch: no word of an earlier one may carry a number
  const int64_t bytes = token_words(a.hid, a.QKVN, a.I, a.H, a.D) * static_cast<int64_t>(sizeof(Word));
  if (cudaMemsetAsync(words, 0, bytes, s) != cudaSuccess || cudaMemsetAsync(a.sync, 0, 16 * sizeof(unsigned int), s) != cudaSuccess)
    return fail(CTDK_ELAUNCH, "decode: clearing the exchange words failed");
  void* params[] = {&a};
  const cudaError_t err = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel_of(a.D, a.tile_bytes)), dim3(grid), dim3(kThreads + 32), params,
                                                      smem, s);
  if (err != cudaSuccess) return fail(CTDK_ELAUNCH, "decode: cooperative launch failed: %s", cudaGetErrorString(err));
  return check_launch("decode token kernel");
}

}  // namespace ctdk
