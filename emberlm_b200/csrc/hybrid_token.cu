// Persistent token kernel of the layer-list family (hybrid_token.h), sandwich layers. Per layer with two branches:
//   [sandwich norms + stacked input projection] | [mix: attention key ranges, recurrent heads]
//   | [branch norms and gates + output projections] | [branch average, norms + gate|up] | [GLU + down]
// and per token the head with the arg-max. A cooperative grid, one CTA per SM, stays resident over all tokens of a
// launch. Weights pass through the ring of token_ring.cuh while the compute warps wait and stage; vectors between phases are
// fp32 behind grid barriers, and every CTA stages (and norms) its own copy. All waits are bounded.
// What bounds a phase (10 000 to 16 000 cycles; its weights would take 3000) is its dependent chain: the barrier (3200 cycles),
// the norms (2500 to 3500 at widths up to 2048; wider ones walk the columns several times) or the merging of the key ranges
// (7400), the products (800 a turn), the mix items (10 000).
// zutalix-0.6b, 300 + 64 tokens: 109.4 -> 64.5 ms against sixteen warps that took the rows from L2 and the items' inputs behind
// the barrier. The items' keys, states and gate rows are on their way before it now, and a phase's description one phase ahead.
#include <cfloat>

#include "decode_core.h"
#include "mma_bf16.cuh"
#include "token_common.cuh"
#include "token_ring.cuh"

namespace ctdk {
namespace hybrid {
namespace {

// 16-byte chunks of a lane in a piece: 32 values of the vector in registers.
template <typename T>
constexpr int kTokenLaneChunks = 2 * sizeof(T);

template <int N>
__device__ __forceinline__ void block_sum(float (&v)[N], float* red /* [N][kRingWarps] */) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  ring_sync();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    v[k] = warp_sum(v[k]);
    if (lane == 0) red[k * kRingWarps + wid] = v[k];
  }
  ring_sync();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < kRingWarps; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(red + k * kRingWarps + i);
      t += (f.x + f.y) + (f.z + f.w);
    }
    v[k] = t;
  }
}

// xs[0, width) = the normed input of a projection but for the last norm's factor, which is returned (the product's rows are
// multiplied by it); CTA 0 stores the new residual. Zero padding to a multiple of 8. A thread keeps to its own columns: Q
// turns of V neighbouring ones are requested at once with their norm weights, so that the chain is one trip to L2 and two or
// three sums. V = 1 takes any width, turn by turn where Q = 0.
template <typename T, int V, int Q>
__device__ __forceinline__ float stage_norm(const TokenArgs& a, const TokenPhase& ph, int64_t tok, float* xs, float* red) {
  constexpr int kStep = V * kRingThreads, kQ = Q > 0 ? Q : 1;
  const int W = a.width, tid = threadIdx.x, first_c = V * tid;
  const float inv = 1.0f / static_cast<float>(W);
  const bool two = ph.y2 != nullptr, first = ph.first_token != 0, known = known_id(a, tok);
  const T* e = static_cast<const T*>(a.embed) + (first && known ? tok * a.ld_embed : 0);
  const float* w_post = first ? a.w_embed : ph.w_post;
  const bool store = blockIdx.x == 0 && ph.x_out != nullptr;
  Cols<V> y[kQ], y2[kQ], wy[kQ], wy2[kQ], x[kQ], wp[kQ], wn[kQ];
  auto sublayer = [&](int u, int c) {   // requests
    if (first) y[u].get(e + c);
    else y[u].load(ph.y + c);
    if (two) y2[u].load(ph.y2 + c);
  };
  auto rest = [&](int u, int c) {
    if (two) {
      wy[u].get(ph.w_y + c);
      wy2[u].get(ph.w_y2 + c);
    }
    if (!first) x[u].load(ph.x + c);
    wp[u].get(w_post + c);
    wn[u].get(ph.w_pre + c);
  };
  auto each = [&](auto f) {
    if constexpr (Q > 0) {
#pragma unroll
      for (int u = 0; u < Q; ++u)
        if (first_c + u * kStep < W) f(u, first_c + u * kStep);
    } else {
#pragma unroll 1
      for (int c = first_c; c < W; c += kStep) f(0, c);
    }
  };
  if constexpr (Q > 0) {
    each(sublayer);
    each(rest);
  }
  float s1 = 1.0f, s2 = 0.0f;
  if (two) {
    float ss[2] = {0.0f, 0.0f};
    each([&](int u, int c) {
      if constexpr (Q == 0) sublayer(u, c);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        ss[0] += y[u].v[k] * y[u].v[k];
        ss[1] += y2[u].v[k] * y2[u].v[k];
      }
    });
    block_sum(ss, red);
    s1 = rsqrtf(ss[0] * inv + a.eps);
    s2 = rsqrtf(ss[1] * inv + a.eps);
  }
  float sum[1] = {0.0f};
  auto combined = [&](int u, int k) {   // a sublayer's result
    if (first) return known ? y[u].v[k] : 0.0f;
    return two ? 0.5f * (y[u].v[k] * s1 * wy[u].v[k] + y2[u].v[k] * s2 * wy2[u].v[k]) : y[u].v[k];
  };
  each([&](int u, int c) {
    if constexpr (Q == 0) {
      sublayer(u, c);
      rest(u, c);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      y[u].v[k] = combined(u, k);
      sum[0] += y[u].v[k] * y[u].v[k];
    }
    if constexpr (Q == 0) y[u].put(xs + c);
  });
  block_sum(sum, red);
  const float sc = rsqrtf(sum[0] * inv + a.eps);
  sum[0] = 0.0f;
  each([&](int u, int c) {
    if constexpr (Q == 0) {
      rest(u, c);
      y[u].get(xs + c);
    }
    Cols<V> n;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float v = (first ? 0.0f : x[u].v[k]) + y[u].v[k] * sc * wp[u].v[k];
      sum[0] += v * v;
      y[u].v[k] = v;
      n.v[k] = v * wn[u].v[k];
    }
    n.put(xs + c);
    if (store) y[u].put(ph.x_out + c);
  });
  if (tid < 8 && W + tid < ((W + 7) & ~7)) xs[W + tid] = 0.0f;
  block_sum(sum, red);   // its barriers also publish xs
  return rsqrtf(sum[0] * inv + a.eps);
}

// Key ranges in use at a slot of the chunk, and their length: of 16 keys, as many as leave all of the phase's items one turn of the CTAs
// (br.splits), more of them where the ranges would be longer than kRangeMost: a second item, a recurrent one, costs a CTA as much as
// about 60 keys. Eight layers of width 2048 with 8 key/value heads, chunks of 8192, us a token behind 1000 and 8000 positions: with
// 32 recurrent heads (4 ranges at least) 827 -> 711 and 2457 -> 1095, with 16 (10 ranges) 588 -> 585 and 1256 -> 991.
constexpr int kRangeMost = 128;
__device__ __forceinline__ int attention_ranges(const TokenBranch& br, int slot, int& per) {
  const int L = slot + 1, n = max(min(br.splits, (L + 15) / 16), min(kAttnSplits, (L + kRangeMost - 1) / kRangeMost));
  per = quotient(L + n - 1, n);
  return quotient(L + per - 1, per);
}

// Outputs of the mix phase as inputs of the output projections; scale: what the rows of a branch's product are
// multiplied by; ranges: key ranges that the mix phase used.
__device__ __forceinline__ void stage_mixed(const TokenArgs& a, const TokenPhase& ph, int ranges, float* sm, float* red, float (&scale)[2]) {
  float ss[2] = {0.0f, 0.0f};
  scale[0] = scale[1] = 1.0f;
  for (int b = 0; b < ph.n_branch; ++b) {
    const TokenBranch& br = ph.br[b];
    float* xs = sm + br.stage_at;
    const int n = br.H * br.vdim;
    if (br.kind == kTokAttention) {   // merges the key ranges: a warp per head, a lane per range, then per four columns
      const int stride = br.dim + kAttnStats, lane = threadIdx.x & 31;
      const bool vec = (br.dim & 3) == 0;
#pragma unroll 1
      for (int h = threadIdx.x >> 5; h < br.H; h += kRingWarps) {
        const float* part = br.part + static_cast<int64_t>(h) * kAttnSplits * stride;
        const float gate = ldg_f(ph.proj + br.col_g + h);
        const float m = lane < ranges ? ldg_f(part + lane * stride) : -FLT_MAX, l = lane < ranges ? ldg_f(part + lane * stride + 1) : 0.0f;
        float w = 0.0f;
#pragma unroll 1
        for (int c0 = 0; c0 < br.dim; c0 += 128) {
          const int c = c0 + 4 * lane;
          const float* of = part + kAttnStats + (c < br.dim ? c : 0);
          float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
          for (int r0 = 0; r0 < ranges; r0 += 8) {
            float4 v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              v[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
              if (r0 + r >= ranges) continue;
              const float* at = of + (r0 + r) * stride;
              if (vec) v[r] = ldg4(at);
              else v[r] = make_float4(ldg_f(at), c + 1 < br.dim ? ldg_f(at + 1) : 0.0f, c + 2 < br.dim ? ldg_f(at + 2) : 0.0f, c + 3 < br.dim ? ldg_f(at + 3) : 0.0f);
            }
            if (c0 == 0 && r0 == 0) {
              const float most = warp_max(m);
              w = lane < ranges ? expf(m - most) : 0.0f;
              w *= sigmoid_f(gate) / warp_sum(w * l);
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const float f = __shfl_sync(0xffffffffu, w, r0 + r);
              o = make_float4(fmaf(f, v[r].x, o.x), fmaf(f, v[r].y, o.y), fmaf(f, v[r].z, o.z), fmaf(f, v[r].w, o.w));
            }
          }
          float* to = xs + h * br.dim + c;
          if (c < br.dim) to[0] = o.x;
          if (c + 1 < br.dim) to[1] = o.y;
          if (c + 2 < br.dim) to[2] = o.z;
          if (c + 3 < br.dim) to[3] = o.w;
        }
      }
    } else if (br.kind == kTokLightning) {   // the norm's factor is the scale
      float t = 0.0f;
      const float* g = ph.proj + br.col_g;
      if (((n | br.col_g) & 3) == 0) {
#pragma unroll 1
        for (int i = 4 * threadIdx.x; i < n; i += 4 * kRingThreads) {
          const float4 v = ldg4(br.out + i), z = ldg4(g + i), w = load4(br.w_norm + i);
          t += sq4(v);
          store4(xs + i, make_float4(v.x * w.x * sigmoid_f(z.x), v.y * w.y * sigmoid_f(z.y), v.z * w.z * sigmoid_f(z.z), v.w * w.w * sigmoid_f(z.w)));
        }
      } else {
#pragma unroll 1
        for (int i = threadIdx.x; i < n; i += kRingThreads) {
          const float v = ldg_f(br.out + i);
          t += v * v;
          xs[i] = v * br.w_norm[i] * sigmoid_f(ldg_f(g + i));
        }
      }
      ss[b] = t;
    } else {
      const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
      for (int h = wid; h < br.H; h += kRingWarps) {
        constexpr int kHeld = 8;   // 256 columns in registers, the others are read twice
        float v[kHeld], f[kHeld], t = 0.0f;
#pragma unroll
        for (int u = 0; u < kHeld; ++u) {
          const int d = lane + 32 * u;
          v[u] = d < br.vdim ? ldg_f(br.out + h * br.vdim + d) : 0.0f;
          f[u] = d < br.vdim ? br.w_norm[d] * sigmoid_f(ldg_f(br.gate + h * br.vdim + d)) : 0.0f;
          t += v[u] * v[u];
        }
        for (int d = lane + 32 * kHeld; d < br.vdim; d += 32) {
          const float w = ldg_f(br.out + h * br.vdim + d);
          t += w * w;
        }
        t = warp_sum(t);   // behind the loop: its trips differ between the lanes
        const float sc = rsqrtf(t / static_cast<float>(br.vdim) + a.eps);
#pragma unroll
        for (int u = 0; u < kHeld; ++u)
          if (lane + 32 * u < br.vdim) xs[h * br.vdim + lane + 32 * u] = v[u] * sc * f[u];
        for (int d = lane + 32 * kHeld; d < br.vdim; d += 32)
          xs[h * br.vdim + d] = ldg_f(br.out + h * br.vdim + d) * sc * br.w_norm[d] * sigmoid_f(ldg_f(br.gate + h * br.vdim + d));
      }
    }
    if (threadIdx.x < 8 && n + threadIdx.x < ((n + 7) & ~7)) xs[n + threadIdx.x] = 0.0f;
  }
  block_sum(ss, red);   // its barriers also publish the vectors
  for (int b = 0; b < ph.n_branch; ++b)
    if (ph.br[b].kind == kTokLightning) scale[b] = rsqrtf(ss[b] / static_cast<float>(ph.br[b].H * ph.br[b].vdim) + a.eps);
}

// ---- items of the mix phase ----
// What an item reads that does not depend on the token (cached keys and their angles, states, low-rank rows) is copied to
// shared memory while the CTA waits for the projections, request_item(), for the CTA's first item. Which item that is takes
// half a dozen divisions, which are made there too.
struct MixItem {
  int branch;      // -1: none
  int head, part;  // attention: key/value head and range; recurrences: head and block of 32 columns
  int slot, j0, j1; // attention: slot of this position, slots of the range
  int ranges;      // of the phase's attention branch, set for every CTA, as is the number of
  int items;       // all items of the phase
  int group;       // delta: head of the queries and keys
  int tap;         // delta: place of this position in the ring of the convolutions
};
__device__ __forceinline__ MixItem mix_item(const TokenPhase& ph, int it, int pos) {
  MixItem m{-1, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int b = 0; b < ph.n_branch; ++b) {
    const TokenBranch& br = ph.br[b];
    int n = br.items;
    if (br.kind == kTokAttention) {
      int per;
      m.slot = pos < br.chunk ? pos : pos % br.chunk;
      m.ranges = attention_ranges(br, m.slot, per);
      n = br.G * m.ranges;
      if (it >= 0 && it < n) {
        m.branch = b;
        m.part = quotient(it, br.G);
        m.head = it - m.part * br.G;
        m.j0 = m.part * per;
        m.j1 = min(m.slot + 1, m.j0 + per);
      }
    } else if (it >= 0 && it < n) {
      const int nb = (br.vdim + 31) / 32;
      m.branch = b;
      m.head = quotient(it, nb);
      m.part = it - m.head * nb;
      if (br.kind == kTokDelta) {
        m.group = quotient(m.head, br.group);
        m.tap = pos - quotient(pos, br.taps) * br.taps;
      }
    }
    it -= n;
    m.items += n;
  }
  return m;
}

// n 16-byte pieces dealt to the block.
__device__ __forceinline__ void copy16(void* dst, const void* src, int n) {
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += kRingThreads) cp_async16(static_cast<char*>(dst) + 16 * i, static_cast<const char*>(src) + 16 * i);
}
__device__ __forceinline__ void copy_bytes(void* dst, const void* src, int bytes) {   // 2-byte aligned
  if (((reinterpret_cast<uintptr_t>(src) | bytes) & 15) == 0) {
    copy16(dst, src, bytes >> 4);
    return;
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < bytes >> 1; i += kRingThreads)
    static_cast<uint16_t*>(dst)[i] = __ldcg(static_cast<const unsigned short*>(src) + i);
}

template <typename T>
struct KeyTile {
  float2* angles;   // [keys][rot_pairs]
  T* keys;          // [keys][dim]
  __device__ __forceinline__ KeyTile(const TokenBranch& br, float* at) : angles(reinterpret_cast<float2*>(at)) {
    keys = reinterpret_cast<T*>(angles + ((br.tile_keys * br.rot_pairs + 1) & ~1));
  }
  // Slots [j, j + n) of head g.
  __device__ __forceinline__ void request(const TokenBranch& br, int g, int j, int n) {
    copy_bytes(angles, br.table + static_cast<int64_t>(j) * br.rot_pairs, n * br.rot_pairs * 8);
    copy_bytes(keys, static_cast<const T*>(br.cache) + (static_cast<int64_t>(g) * br.chunk + j) * br.dim, n * br.dim * static_cast<int>(sizeof(T)));
    cp_async_commit();
  }
};

// Floats of partial sums: of the warps' shares of the keys, or of the blocks of 32 columns beyond the warps' first ones.
inline int attention_scratch(int dim) { return std::max(kRingWarps * 34, (dim + 32 * kRingWarps - 1) / (32 * kRingWarps) * kRingThreads); }

// The new token against the keys [j0, j1) of key/value head g, all query heads of the group, into the partial results of
// the range. Keys are the values. 16 threads per key for the scores, a warp per 32 columns of a head and share of the keys
// for the sums.
template <typename T>
__device__ __forceinline__ void attention_item(const TokenPhase& ph, const TokenBranch& br, const MixItem it, int pos, float* sm, float* tile_at, bool requested) {
  const int g = it.head, dim = br.dim, P = (dim + 1) >> 1, hq = br.group, KT = br.tile_keys, j0 = it.j0, j1 = it.j1;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, stride = dim + kAttnStats;
  KeyTile<T> tile(br, tile_at);
  if (!requested) tile.request(br, g, j0, min(KT, j1 - j0));
  float* qs = sm;                    // [hq][2 P] rotated, scaled
  float* kn = qs + hq * 2 * P;       // [2 P] this token's key
  float* sc = kn + 2 * P;            // [hq][32] scores
  float* scr = sc + hq * 32;         // [kRingWarps][34], or a float of every thread and turn (attention_scratch)
  const int slot = it.part == it.ranges - 1 ? j1 - 1 : -1;   // the last range holds the new position
#pragma unroll 1
  for (int r = wid; r < hq + (slot >= 0 ? 1 : 0); r += kRingWarps) {
    const bool key = r == hq;
    const float* src = ph.proj + (key ? br.col_k + g * dim : br.col_q + (g * hq + r) * dim);
    const float* bias = key ? br.b_k + g * dim : br.b_q + (g * hq + r) * dim;
    const float2* angles = br.table + static_cast<int64_t>(it.slot) * br.rot_pairs;
    float* to = key ? kn : qs + r * 2 * P;
    T* row = static_cast<T*>(br.cache) + (static_cast<int64_t>(g) * br.chunk + it.slot) * dim;
#pragma unroll 2
    for (int p = lane; p < P; p += 32) {
      const int d = 2 * p;
      const bool pair = d + 1 < dim;
      const float2 rot = p < br.rot_pairs && !key ? angles[p] : make_float2(1.0f, 0.0f);
      const float u = ldg_f(src + d) + bias[d], v = pair ? ldg_f(src + d + 1) + bias[d + 1] : 0.0f;
      const float f = key ? 1.0f : br.scale;
      *reinterpret_cast<float2*>(to + d) = make_float2((u * rot.x - v * rot.y) * f, (v * rot.x + u * rot.y) * f);
      if (key) {
        row[d] = from_f<T>(u);
        if (pair) row[d + 1] = from_f<T>(v);
      }
    }
  }
  const int nb = (dim + 31) >> 5, at_once = nb == 1 ? 8 : (nb == 2 ? 4 : (nb <= 4 ? 2 : 1));   // kRingWarps / nb
#pragma unroll 1
  for (int g0 = 0; g0 < hq; g0 += at_once) {
    // blocks of 32 columns, a warp each, with shares of the keys where there are more warps; of a head with more blocks than
    // warps every warp takes several, whose sums stand in `scr` between two tiles
    const int heads = min(at_once, hq - g0), blocks = heads * nb, turns = (blocks + kRingWarps - 1) / kRingWarps;
    const int sh = blocks * 8 <= kRingWarps ? 3 : (blocks * 4 <= kRingWarps ? 2 : (blocks * 2 <= kRingWarps ? 1 : 0)), shares = 1 << sh;
    int blk = wid, share = 0, h = g0;
    if (turns == 1) {
#pragma unroll 1
      for (; blk >= blocks; blk -= blocks) ++share;
#pragma unroll 1
      for (; blk >= nb; blk -= nb) ++h;   // blk: block of the head's columns
    }
    const bool takes_part = share < shares;
    float m = -FLT_MAX, l = 0.0f, o = 0.0f;
#pragma unroll 1
    for (int jb = j0; jb < j1; jb += KT) {
      const int n = min(KT, j1 - jb);
      if (jb != j0 || g0 > 0) {
        ring_sync();   // the tile has been read
        if (j1 - j0 > KT) tile.request(br, g, jb, n);
      }
      cp_async_wait<0>();
      ring_sync();
      const int t = threadIdx.x & 15;
#pragma unroll 1
      for (int key = threadIdx.x >> 4; key < 32; key += kRingThreads / 16) {
        const bool fresh = jb + key == slot;
#pragma unroll 1
        for (int h0 = g0; h0 < g0 + heads; h0 += 4) {
          float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (key < n) {
#pragma unroll 1
            for (int p = t; p < P; p += 16) {
              const int d = 2 * p;
              const T* row = tile.keys + key * dim + d;
              const float u = fresh ? kn[d] : to_f(row[0]), v = fresh ? kn[d + 1] : (d + 1 < dim ? to_f(row[1]) : 0.0f);
              const float2 rot = p < br.rot_pairs ? tile.angles[key * br.rot_pairs + p] : make_float2(1.0f, 0.0f);
              const float x = u * rot.x - v * rot.y, y = v * rot.x + u * rot.y;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 q = *reinterpret_cast<const float2*>(qs + min(h0 + k, hq - 1) * 2 * P + d);
                acc[k] = fmaf(q.x, x, fmaf(q.y, y, acc[k]));
              }
            }
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], x);
            if (t == 0 && h0 + k < g0 + heads) sc[(h0 + k) * 32 + key] = acc[k];
          }
        }
      }
      ring_sync();
      if (takes_part) {
        const int mine = (n - share + shares - 1) >> sh;   // keys share, share + shares, ... of the tile
        const float d = lane < mine ? sc[h * 32 + share + lane * shares] : -FLT_MAX;
        const float most = fmaxf(m, warp_max(d)), w = lane < mine ? expf(d - most) : 0.0f, fix = expf(m - most);
        m = most;
        l = l * fix + warp_sum(w);
#pragma unroll 1
        for (int turn = 0; turn < turns; ++turn) {
          const int col = (blk + turn * kRingWarps) * 32 + lane, c = col < dim ? col : 0;
          if (turns > 1 && jb != j0) o = scr[turn * kRingThreads + threadIdx.x];
          o *= fix;
#pragma unroll 4
          for (int i = 0; i < mine; ++i) {
            const int key = share + i * shares;
            const float v = jb + key == slot ? kn[c] : to_f(tile.keys[key * dim + c]);
            o = fmaf(__shfl_sync(0xffffffffu, w, i), v, o);
          }
          if (turns > 1) {
            scr[turn * kRingThreads + threadIdx.x] = o;
            o = 0.0f;
          }
        }
      }
    }
    if (shares > 1) {
      if (takes_part) {
        scr[wid * 34 + 2 + lane] = o;
        if (lane == 0) *reinterpret_cast<float2*>(scr + wid * 34) = make_float2(m, l);
      }
      ring_sync();
      if (takes_part && share == 0) {
#pragma unroll 1
        for (int k = 1; k < shares; ++k) {
          const float* other = scr + (wid + k * blocks) * 34;
          const float most = fmaxf(m, other[0]), f = expf(m - most), fo = expf(other[0] - most);
          l = l * f + other[1] * fo;
          o = o * f + other[2 + lane] * fo;
          m = most;
        }
      }
    }
    if (takes_part && share == 0) {
      float* dst = br.part + (static_cast<int64_t>(g * hq + h) * kAttnSplits + it.part) * stride;
#pragma unroll 1
      for (int turn = 0; turn < turns; ++turn) {
        const int col = (blk + turn * kRingWarps) * 32 + lane;
        if (turns > 1) o = scr[turn * kRingThreads + threadIdx.x];   // of this thread
        if (col < dim) dst[kAttnStats + col] = o;
      }
      if (blk == 0 && lane == 0) {
        dst[0] = m;
        dst[1] = l;
      }
    }
  }
}

// Sum over the warps of a per-lane value; every thread gets its lane's total. red: read until the next call but one.
__device__ __forceinline__ float column_sum(float v, float* red /* [kRingWarps][32] */) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  red[wid * 32 + lane] = v;
  ring_sync();
  float t = 0.0f;
#pragma unroll
  for (int i = 0; i < kRingWarps; ++i) t += red[i * 32 + lane];
  return t;
}

// Columns [c0, c0 + 32) of a head's state, rows of 32 floats.
__device__ __forceinline__ void request_state(float* tile, const float* S, int dim, int vdim, int c0) {
  if ((vdim & 3) == 0) {
    const int quads = min(8, (vdim - c0) >> 2);
#pragma unroll 1
    for (int i = threadIdx.x; i < dim * 8; i += kRingThreads) {
      const int r = i >> 3, q = i & 7;
      if (q < quads) cp_async16(tile + r * 32 + 4 * q, S + static_cast<int64_t>(r) * vdim + c0 + 4 * q);
    }
  } else {
    const int cols = min(32, vdim - c0);
#pragma unroll 1
    for (int i = threadIdx.x; i < dim * 32; i += kRingThreads)
      if ((i & 31) < cols) tile[i] = ldg_f(S + static_cast<int64_t>(i >> 5) * vdim + c0 + (i & 31));
  }
}

// 32 value columns of one lightning head: a lane per column, the key rows dealt to the warps.
__device__ __forceinline__ void lightning_item(const TokenPhase& ph, const TokenBranch& br, const MixItem it, int pos, float* sm, float* tile, bool requested) {
  const int h = it.head, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = it.part * 32 + lane, dim = br.dim;
  float *q = sm, *k = q + dim, *red = k + dim;
  float* S = br.state + static_cast<int64_t>(h) * dim * br.vdim + c;
  if (!requested && pos > 0) {
    request_state(tile, br.state + static_cast<int64_t>(h) * dim * br.vdim, dim, br.vdim, c - lane);
    cp_async_commit();
  }
  const bool live = c < br.vdim;
  const float v = live ? silu_f(ldg_f(ph.proj + br.col_v + h * br.vdim + c)) : 0.0f, dec = br.decay[h];
#pragma unroll 1
  for (int d = threadIdx.x; d < 2 * dim; d += kRingThreads)
    q[d] = silu_f(ldg_f(ph.proj + (d < dim ? br.col_q + d : br.col_k + d - dim) + h * dim));
  cp_async_wait<0>();
  ring_sync();
  float o = 0.0f;
  if (live) {
#pragma unroll 4
    for (int r = wid; r < dim; r += kRingWarps) {
      const float s1 = fmaf(dec, pos > 0 ? tile[r * 32 + lane] : 0.0f, k[r] * v);
      S[static_cast<int64_t>(r) * br.vdim] = s1;
      o = fmaf(s1, q[r], o);
    }
  }
  o = column_sum(o, red);
  if (wid == 0 && live) br.out[h * br.vdim + c] = o;
}

// This token's value of convolution channel (ring channel rc, stacked projection column col), activated. tap: pos mod taps.
__device__ __forceinline__ float conv_channel(const TokenPhase& ph, const TokenBranch& br, int pos, int tap, int col, const float* taps, int rc,
                                              int ring_ld, bool owner) {
  const float now = ldg_f(ph.proj + col);
  const int n = br.taps;
  float y = 0.0f;
#pragma unroll 4
  for (int j = 0; j < n - 1; ++j) {   // position pos - (n - 1) + j
    const int at = tap + 1 + j < n ? tap + 1 + j : tap + 1 + j - n;
    if (pos - (n - 1) + j >= 0) y = fmaf(taps[j], ldg_f(br.ring + static_cast<int64_t>(at) * ring_ld + rc), y);
  }
  // the slot being overwritten is taps positions old: nobody reads it for this token
  if (owner) br.ring[static_cast<int64_t>(tap) * ring_ld + rc] = now;
  return silu_f(fmaf(taps[n - 1], now, y));
}

// dot of a low-rank row with a staged fp32 vector (rank rounded up to 8, both zero-padded); 2^log_lanes
// neighbouring threads share a row, `turn` (0 or 1) staggers the rows over the banks. All of them get the sum.
template <typename T>
__device__ __forceinline__ float short_dot(const T* row, const float* x, int n, int log_lanes, int turn) {
  constexpr int N = Chunk<T>::kN;
  float acc = 0.0f;
  const int lanes = 1 << log_lanes, chunks = n / N, rounds = (chunks + lanes - 1) >> log_lanes;
#pragma unroll 2
  for (int i = 0; i < rounds; ++i) {
    const int at = i + turn < rounds ? i + turn : i + turn - rounds;
    const int c = (at << log_lanes) + (static_cast<int>(threadIdx.x) & (lanes - 1));
    if (c >= chunks) continue;
    Chunk<T> w;
    w.w = *reinterpret_cast<const decltype(w.w)*>(row + c * N);
    acc = w.dot(x + c * N, acc);
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// Delta rule: the tile of the state [dim][32], then the head's low-rank rows of the decays and of the columns' gates, if
// they fit.
template <typename T>
struct DeltaTile {
  float* state;
  T *a2, *g2;
  const T *a2_from, *g2_from;
  int a2_bytes, g2_bytes;
  __device__ __forceinline__ DeltaTile(const TokenBranch& br, const MixItem& it, float* at) : state(at) {
    const int h = it.head, c0 = it.part * 32, ra = (br.rank_a + 7) & ~7, rg = (br.rank_g + 7) & ~7;
    a2 = reinterpret_cast<T*>(at + br.dim * 32);
    a2_bytes = br.dim * ra * static_cast<int>(sizeof(T));
    g2 = a2 + br.dim * ra;
    g2_bytes = min(32, br.vdim - c0) * rg * static_cast<int>(sizeof(T));
    a2_from = static_cast<const T*>(br.w_a2) + static_cast<int64_t>(h) * br.dim * ra;
    g2_from = static_cast<const T*>(br.w_g2) + (static_cast<int64_t>(h) * br.vdim + c0) * rg;
  }
  __device__ __forceinline__ void request_rows(const TokenBranch& br, const MixItem& it, int pos) {
    if (pos > 0) request_state(state, br.state + static_cast<int64_t>(it.head) * br.dim * br.vdim, br.dim, br.vdim, it.part * 32);
  }
  __device__ __forceinline__ void request(const TokenBranch& br, const MixItem& it, int pos) {
    if (!br.state_late) request_rows(br, it, pos);
    if (br.low_staged) {
      copy16(a2, a2_from, a2_bytes >> 4);
      copy16(g2, g2_from, g2_bytes >> 4);
    }
    cp_async_commit();
  }
};

// 32 value columns of one delta-rule head: a lane per column, the key rows dealt to the warps.
template <typename T>
__device__ __forceinline__ void delta_item(const TokenPhase& ph, const TokenBranch& br, const MixItem it, int pos, float* sm, float* tile_at, bool requested) {
  const int h = it.head, vb = it.part, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int dim = br.dim, grp = it.group, c = vb * 32 + lane;
  const int qk = br.G * dim, ring_ld = 2 * qk + br.H * br.vdim;
  const int ra = (br.rank_a + 7) & ~7, rg = (br.rank_g + 7) & ~7;
  float *a1 = sm, *g1 = a1 + ra, *q = g1 + rg, *k = q + dim, *vs = k + dim, *g = vs + 32, *red = g + dim, *sq = red + 2 * kRingWarps * 32;
  DeltaTile<T> tile(br, it, tile_at);
  if (!requested) tile.request(br, it, pos);
  const bool own_qk = h == grp * br.group && vb == 0, live = c < br.vdim;
  const float beta = sigmoid_f(ldg_f(ph.proj + br.col_b + h)), amp = -expf(br.a_log[h]);
  // staged vectors, in one run of indexes: q, k, v of the columns, then a1 and g1
  float ss[2] = {0.0f, 0.0f};
#pragma unroll 1
  for (int i = threadIdx.x; i < 2 * dim + 32 + ra + rg; i += kRingThreads) {
    if (i < 2 * dim + 32) {
      const bool is_k = i >= dim, is_v = i >= 2 * dim;
      const int d = is_v ? i - 2 * dim : (is_k ? i - dim : i), ch = is_v ? h * br.vdim + vb * 32 + d : grp * dim + d;
      if (is_v && vb * 32 + d >= br.vdim) {
        q[i] = 0.0f;
        continue;
      }
      const float* taps = (is_v ? br.conv_v : (is_k ? br.conv_k : br.conv_q)) + static_cast<int64_t>(ch) * br.taps;
      const float y = conv_channel(ph, br, pos, it.tap, (is_v ? br.col_v : (is_k ? br.col_k : br.col_q)) + ch, taps, (is_v ? 2 * qk : (is_k ? qk : 0)) + ch,
                                   ring_ld, is_v || own_qk);
      q[i] = y;   // k and v follow q
      if (!is_k) ss[0] += y * y;
      else if (!is_v) ss[1] += y * y;
    } else {
      const int e = i - 2 * dim - 32;
      a1[e] = e < ra ? (e < br.rank_a ? ldg_f(ph.proj + br.col_a1 + e) : 0.0f) : (e - ra < br.rank_g ? ldg_f(ph.proj + br.col_g1 + e - ra) : 0.0f);
    }
  }
  ss[0] = warp_sum(ss[0]);
  ss[1] = warp_sum(ss[1]);
  if (lane == 0) {
    sq[wid] = ss[0];
    sq[kRingWarps + wid] = ss[1];
  }
  cp_async_wait<0>();
  ring_sync();
  // decays: four threads a channel
#pragma unroll 1
  for (int d0 = 0; d0 < dim; d0 += kRingThreads / 4) {
    const int d = d0 + (threadIdx.x >> 2);
    const float z = short_dot((br.low_staged ? tile.a2 : tile.a2_from) + static_cast<int64_t>(min(d, dim - 1)) * ra, a1, ra, 2, d & 1);
    if ((threadIdx.x & 3) == 0 && d < dim) g[d] = expf(amp * softplus_f(z + br.dt_bias[h * dim + d]));
  }
  // the columns' output gates: 16 threads a column
#pragma unroll 1
  for (int e = threadIdx.x >> 4; e < 32; e += kRingThreads / 16) {
    const float z = short_dot((br.low_staged ? tile.g2 : tile.g2_from) + static_cast<int64_t>(vb * 32 + e < br.vdim ? e : 0) * rg, g1, rg, 4, 0);
    if ((threadIdx.x & 15) == 0 && vb * 32 + e < br.vdim) br.gate[h * br.vdim + vb * 32 + e] = z;
  }
  ring_sync();
  if (br.state_late) {   // a1 and g1 have been read
    tile.state = a1;
    tile.request_rows(br, it, pos);
    cp_async_commit();
    cp_async_wait<0>();
    ring_sync();
  }
  float nq = 0.0f, nk = 0.0f;
#pragma unroll
  for (int i = 0; i < kRingWarps; ++i) {
    nq += sq[i];
    nk += sq[kRingWarps + i];
  }
  const float fq = rsqrtf(nq + 1e-6f) * rsqrtf(static_cast<float>(dim)), fk = rsqrtf(nk + 1e-6f);
  float p = 0.0f;
#pragma unroll 4
  for (int r = wid; r < dim; r += kRingWarps) {
    const float s = pos > 0 && live ? tile.state[r * 32 + lane] * g[r] : 0.0f;
    tile.state[r * 32 + lane] = s;
    p = fmaf(s, k[r] * fk, p);
  }
  const float u = beta * (vs[lane] - column_sum(p, red));
  float* S = br.state + static_cast<int64_t>(h) * dim * br.vdim + c;
  float o = 0.0f;
#pragma unroll 4
  for (int r = wid; r < dim; r += kRingWarps) {
    const float s = fmaf(k[r] * fk, u, tile.state[r * 32 + lane]);
    if (live) S[static_cast<int64_t>(r) * br.vdim] = s;
    o = fmaf(s, q[r] * fq, o);
  }
  o = column_sum(o, red + kRingWarps * 32);
  if (wid == 0 && live) br.out[h * br.vdim + c] = o;
}

template <typename T>
__device__ __forceinline__ MixItem request_item(const TokenPhase& ph, int pos, float* tile_at) {
  const MixItem it = mix_item(ph, blockIdx.x, pos);
  if (it.branch < 0) return it;
  const TokenBranch& br = ph.br[it.branch];
  if (br.kind == kTokAttention) {
    KeyTile<T>(br, tile_at).request(br, it.head, it.j0, min(br.tile_keys, it.j1 - it.j0));
  } else if (br.kind == kTokLightning) {
    if (pos > 0) request_state(tile_at, br.state + static_cast<int64_t>(it.head) * br.dim * br.vdim, br.dim, br.vdim, it.part * 32);
    cp_async_commit();
  } else {
    DeltaTile<T>(br, it, tile_at).request(br, it, pos);
  }
  return it;
}
template <typename T>
__device__ __forceinline__ void mix_phase(const TokenPhase& ph, MixItem it, int pos, float* sm, float* tile_at) {
#pragma unroll 1
  for (int n = blockIdx.x; it.branch >= 0;) {
    const TokenBranch& br = ph.br[it.branch];
    const bool first = n == static_cast<int>(blockIdx.x);
    if (br.kind == kTokAttention) attention_item<T>(ph, br, it, pos, sm, tile_at, first);
    else if (br.kind == kTokLightning) lightning_item(ph, br, it, pos, sm, tile_at, first);
    else delta_item<T>(ph, br, it, pos, sm, tile_at, first);
    n += gridDim.x;
    if (n >= it.items) return;
    it = mix_item(ph, n, pos);
    ring_sync();
  }
}

// The plain products of a phase, out of the ring; scale: of the first one's rows, of the others'. Returns the best arg-max
// key of the head's rows.
template <typename T>
__device__ __forceinline__ unsigned long long plain_products(const TokenPhase& ph, const float* sm, Ring& ring, const float (&scale)[2]) {
  unsigned long long best = 0ull;
  const int v = blockIdx.x;
#pragma unroll 1
  for (int i = 0; i < ph.n_gemv; ++i) {
    const TokenGemv& g = ph.gemv[i];
    const int lo = max(v * ph.per, g.base), hi = min(min((v + 1) * ph.per, ph.plain_rows), g.base + g.rows);
    const float f = i == 0 ? scale[0] : scale[1];
    if (hi <= lo) continue;
    // a wait that ran out is seen at the barrier
    ring_multiply<T, kTokenLaneChunks<T>>(ring, g.ring, hi - lo, false, sm + g.in, [&](int r, float y, float) {
      y *= f;
      const int row = lo - g.base + r;
      g.y[row] = y;
      if (ph.is_head) {
        const unsigned long long k = argmax_key(y, row);
        best = k > best ? k : best;
      }
    });
  }
  return best;
}

// Weights that the items of a coming phase read, into L2.
__device__ __forceinline__ void ask_items(const TokenPhase& ph) {
#pragma unroll 1
  for (int k = 0; k < kMaxAsks; ++k) {
    const char* base = static_cast<const char*>(ph.ask[k]);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * kRingThreads + threadIdx.x; i < ph.ask_bytes[k] / 128; i += static_cast<int64_t>(gridDim.x) * kRingThreads)
      prefetch_l2(base + i * 128);
  }
}

// The requesting warp: this CTA's rows of all plain products, for all tokens.
__device__ __forceinline__ void request_weights(const TokenArgs& a, const Ring& ring) {
  RingRequests q(ring);
  for (int t = 0; t < a.n_tokens; ++t) {
    RingProduct p = a.products[0];
    for (int i = 0; i < a.n_products; ++i) {
      const RingProduct next = a.products[i + 1 < a.n_products ? i + 1 : 0];   // on its way under this one's waits
      const int v = blockIdx.x;
      const int lo = max(v * p.per, p.base), hi = min(min((v + 1) * p.per, p.plain_rows), p.base + p.rows);
      if (hi > lo && !q.rows(static_cast<const char*>(p.W), nullptr, lo - p.base, hi - lo, p.ring)) {
        q.give_up();
        return;
      }
      p = next;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kRingThreads + 32, 1) hybrid_token_kernel(const __grid_constant__ TokenArgs a) {
  extern __shared__ __align__(16) float sm[];   // staged vector, or the items' scratch and what is copied ahead of them; then the ring
  __shared__ TokenPhase ph_s[2];
  __shared__ __align__(16) float red[2 * kRingWarps];
  __shared__ unsigned long long best_s[kRingWarps];
  __shared__ MixItem s_mix;
  __shared__ uint64_t s_bar[2 * kRingMaxStages];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  Ring ring(reinterpret_cast<char*>(sm + a.stage_floats), s_bar, a.stages, a.stage_bytes, a.sync, a.status);
  if (threadIdx.x == 0) ring.init();
  __syncthreads();
  if (wid == kRingWarps) {
    request_weights(a, ring);
    return;
  }
  unsigned int epoch = 0;
  int pos = a.counters[0];
  int64_t tok = *a.cur_token;
  if (!known_id(a, tok) && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.status[2], 1);   // later ones are the kernel's own
  unsigned long long* words = reinterpret_cast<unsigned long long*>(a.sync + 128);
  bool alive = true;
  int slot = 0;
  auto fetch = [&](int i, int to) {   // phase descriptions are on their way one phase ahead
    const char* src = reinterpret_cast<const char*>(a.phases + i);
    char* dst = reinterpret_cast<char*>(&ph_s[to]);
    for (int w = threadIdx.x; w < static_cast<int>(sizeof(TokenPhase) / 16); w += kRingThreads) cp_async16(dst + 16 * w, src + 16 * w);
    cp_async_commit();
  };
  fetch(0, 0);
  cp_async_wait<0>();
  ring_sync();
  for (int t = 0; t < a.n_tokens && alive; ++t) {
#pragma unroll 1
    for (int i = 0; i < a.n_phases; ++i) {
      const TokenPhase& ph = ph_s[slot];
      slot ^= 1;
      fetch(i + 1 < a.n_phases ? i + 1 : 0, slot);
      unsigned long long best = 0ull;
      if (ph.is_mix) {
        mix_phase<T>(ph, s_mix, pos, sm, sm + a.item_at);
      } else {
        float scale[2] = {1.0f, 1.0f};
        if (ph.stage == kStageNorm) {
          if ((a.width & 3) == 0 && a.width <= 4 * kRingThreads) scale[0] = stage_norm<T, 4, 1>(a, ph, tok, sm, red);
          else if ((a.width & 3) == 0 && a.width <= 8 * kRingThreads) scale[0] = stage_norm<T, 4, 2>(a, ph, tok, sm, red);
          else scale[0] = stage_norm<T, 1, 0>(a, ph, tok, sm, red);
        } else if (ph.stage == kStageGlu) {
          batched<4>(ph.ffp >> 2, threadIdx.x, kRingThreads, [&](int c) { return Pair4{ldg4(ph.gu + 4 * c), ldg4(ph.gu + ph.ffp + 4 * c)}; },
                     [&](int c, const Pair4& v) {
                       store4(sm + 4 * c, make_float4(clamped_glu_f(v.a.x, v.b.x, ph.limit), clamped_glu_f(v.a.y, v.b.y, ph.limit),
                                                      clamped_glu_f(v.a.z, v.b.z, ph.limit), clamped_glu_f(v.a.w, v.b.w, ph.limit)));
                     });
          ring_sync();
        } else {
          stage_mixed(a, ph, s_mix.ranges, sm, red, scale);
        }
        best = plain_products<T>(ph, sm, ring, scale);
      }
      if (ph.is_head && a.out_tokens != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long k = __shfl_xor_sync(0xffffffffu, best, o);
          best = k > best ? k : best;
        }
        if (lane == 0) best_s[wid] = best;
        ring_sync();
        if (threadIdx.x == 0) {
#pragma unroll
          for (int w = 1; w < kRingWarps; ++w) best = best_s[w] > best ? best_s[w] : best;
          atomicMax(&words[t & 1], best);
        }
      }
      cp_async_wait<0>();
      if (i + 1 == a.n_phases && a.out_tokens == nullptr) break;   // logits are complete at the end of the kernel
      grid_arrive(a.sync, epoch);
      if (ph_s[slot].is_mix) {   // visible behind the arrival's barrier, what is stored here behind the wait's
        const MixItem it = request_item<T>(ph_s[slot], pos, sm + a.item_at);   // the staged vector has been read
        if (threadIdx.x == 0) s_mix = it;
      }
      ask_items(ph);   // in front of the arrival it was 400 cycles of every phase (65.8 ms against 64.5)
      if (!(alive = grid_wait(a.sync, a.status, 91, epoch))) break;
    }
    if (!alive || a.out_tokens == nullptr) break;
    const unsigned long long wv = *reinterpret_cast<volatile unsigned long long*>(&words[t & 1]);
    tok = static_cast<int64_t>(0xFFFFFFFFu - static_cast<unsigned>(wv & 0xFFFFFFFFull));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.out_tokens[a.out_offset + t] = tok;
      words[(t + 1) & 1] = 0ull;   // last read one barrier ago
    }
    pos += 1;
  }
  cp_async_wait<0>();   // a CTA that leaves early may have copies in flight
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.out_tokens != nullptr) {
    a.counters[0] = pos;
    a.counters[1] += a.n_tokens;
    *a.cur_token = tok;
  }
}

}  // namespace

int token_items(TokenPhase* phases, int n, int* tile_at) {
  constexpr int64_t kTile = 64 * 1024;   // of the low-rank rows or of a tile of keys, where they are large
  constexpr int64_t kLateFloats = 52 * 1024;   // with the shortest ring behind it 222 KB; the ranks are then 40 000 and more, a state 8192 floats
  int64_t scratch = 0, tile = 0;
  for (int i = 0; i < n; ++i) {
    for (int b = 0; b < phases[i].n_branch; ++b) {
      TokenBranch& br = phases[i].br[b];
      br.group = br.G > 0 ? br.H / br.G : 1;
      const int64_t ra = (br.rank_a + 7) & ~7, rg = (br.rank_g + 7) & ~7, size = br.elem;
      int64_t f, t;   // floats, bytes
      if (br.kind == kTokAttention) {
        const int64_t hq = br.H / br.G, key = br.dim * size + br.rot_pairs * 8;
        for (br.tile_keys = 32; br.tile_keys > 1 && br.tile_keys * key > kTile; br.tile_keys /= 2) {
        }
        f = (hq + 1) * (br.dim + 1) + hq * 32 + attention_scratch(br.dim) + 2;
        t = br.tile_keys * key + 32;
      } else if (br.kind == kTokLightning) {
        f = 2 * br.dim + kRingWarps * 32;
        t = br.dim * 128;
      } else {
        f = ra + rg + 3 * br.dim + 32 + 2 * kRingWarps * 32 + 2 * kRingWarps;
        const int64_t low = (br.dim * ra + 32 * rg) * size;
        br.low_staged = low <= kTile ? 1 : 0;
        // the largest ranks leave the state no room of its own and are larger than it
        br.state_late = f + br.dim * 32 > kLateFloats ? 1 : 0;
        t = (br.state_late ? 0 : br.dim * 128) + (br.low_staged ? low : 0);
      }
      scratch = std::max(scratch, f);
      tile = std::max(tile, (t + 127) / 128 * 32);
    }
  }
  *tile_at = static_cast<int>((scratch + 31) / 32 * 32);
  return *tile_at + static_cast<int>(tile);
}

// Pieces of up to kTokenLaneChunks chunks a lane, less where that does not leave room for three stages.
template <typename T>
size_t token_plan(TokenPhase* phases, int n, int grid, TokenArgs& a, std::vector<RingProduct>& products) {
  // The kernel's own arrays come on top. 64 KB stay L1, where the stack lives, unless the staged vector is so large that no ring
  // fits: zutalix-0.6b's 300 + 64 tokens take 64.7 ms so, 66.8 with all of it for the ring, 87 with 100 KB in all.
  constexpr int64_t kOwn = 6144;
  static_assert(2 * sizeof(TokenPhase) + 1024 <= kOwn, "shared memory");
  a.stage_floats = (a.stage_floats + 31) / 32 * 32;
  for (int step = 0; step < 12; ++step) {
    const int piece = (32 * kTokenLaneChunks<T>) >> (step % 6);
    const int64_t room = (step < 6 ? 164 : 227) * 1024 - kOwn;
    if (piece < 16) continue;
    products.clear();
    a.stage_bytes = 256;
    for (int i = 0; i < n; ++i) {
      TokenPhase& p = phases[i];
      p.plain_rows = 0;
      for (int k = 0; k < p.n_gemv; ++k) {
        p.gemv[k].base = p.plain_rows;
        p.plain_rows += p.gemv[k].rows;
      }
      p.per = ceil_div(p.plain_rows, grid);
      for (int k = 0; k < p.n_gemv; ++k) {
        TokenGemv& g = p.gemv[k];
        g.ring = ring_rows(g.K * static_cast<int>(sizeof(T)) / 16, piece);
        a.stage_bytes = std::max(a.stage_bytes, ring_stage_bytes(g.ring));
        products.push_back(RingProduct{g.W, g.rows, g.base, p.per, p.plain_rows, g.ring});
      }
    }
    a.stages = static_cast<int>(std::min<int64_t>((room - a.stage_floats * 4) / a.stage_bytes, kRingMaxStages));
    if (a.stages >= 3) break;
  }
  a.n_products = static_cast<int>(products.size());
  return a.stages >= 3 ? static_cast<size_t>(a.stage_floats) * 4 + static_cast<size_t>(a.stages) * a.stage_bytes : 0;
}

template <typename T>
int token_grid(size_t smem, int* grid) {
  return cooperative_grid(reinterpret_cast<const void*>(hybrid_token_kernel<T>), kRingThreads + 32, smem, grid);
}

template <typename T>
int launch_token_kernel(const TokenArgs& a, int grid, size_t smem, cudaStream_t s) {
  return cooperative_launch(reinterpret_cast<const void*>(hybrid_token_kernel<T>), a, grid, kRingThreads + 32, smem, s);
}

int cooperative_grid(const void* kernel, int threads, size_t smem, int* grid) {
  int dev = 0, coop = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (e == cudaSuccess) e = raise_dynamic_smem(kernel, smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (e != cudaSuccess) return fail(CTDK_ELAUNCH, "hybrid token kernel: %s", cudaGetErrorString(e));
  CTDK_REQUIRE(coop != 0 && per_sm >= 1, "hybrid token kernel: no cooperative launch with %zu bytes of shared memory", smem);
  *grid = sm_count();
  return CTDK_OK;
}
int cooperative_launch(const void* kernel, const TokenArgs& a, int grid, int threads, size_t smem, cudaStream_t s) {
  if (cudaMemsetAsync(a.sync, 0, a.sync_words * sizeof(unsigned int), s) != cudaSuccess)
    return fail(CTDK_ELAUNCH, "hybrid token kernel: clearing the barrier words failed");
  TokenArgs args = a;
  void* params[] = {&args};
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), params, smem, s);
  if (e != cudaSuccess) return fail(CTDK_ELAUNCH, "hybrid token kernel: %s", cudaGetErrorString(e));
  return check_launch("hybrid token kernel");
}

template size_t token_plan<float>(TokenPhase*, int, int, TokenArgs&, std::vector<RingProduct>&);
template size_t token_plan<__nv_bfloat16>(TokenPhase*, int, int, TokenArgs&, std::vector<RingProduct>&);
template int token_grid<float>(size_t, int*);
template int token_grid<__nv_bfloat16>(size_t, int*);
template int launch_token_kernel<float>(const TokenArgs&, int, size_t, cudaStream_t);
template int launch_token_kernel<__nv_bfloat16>(const TokenArgs&, int, size_t, cudaStream_t);

}  // namespace hybrid
}  // namespace ctdk
