// What the token kernels of the layer-list family share: chunks of weights, batched loads, neighbouring columns.
#pragma once

#include "hybrid_kernels.h"
#include "hybrid_token.h"

namespace ctdk {
namespace hybrid {

__device__ __forceinline__ float ldg_f(const float* p) { return __ldcg(p); }

// Eight (bfloat16) or four (fp32) weights, from memory, against the vector in shared memory (RingChunk of token_ring.cuh: from
// shared memory against values that a lane holds).
template <typename T>
struct Chunk;
template <>
struct Chunk<float> {
  static constexpr int kN = 4;
  float4 w;
  __device__ __forceinline__ void load(const float* p) { w = __ldcs(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ float dot(const float* x, float acc) const {
    const float4 v = *reinterpret_cast<const float4*>(x);
    acc = fmaf(w.x, v.x, acc);
    acc = fmaf(w.y, v.y, acc);
    acc = fmaf(w.z, v.z, acc);
    return fmaf(w.w, v.w, acc);
  }
  __device__ __forceinline__ void unpack(float (&o)[4]) const {
    o[0] = w.x;
    o[1] = w.y;
    o[2] = w.z;
    o[3] = w.w;
  }
};
template <>
struct Chunk<__nv_bfloat16> {
  static constexpr int kN = 8;
  uint4 w;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { w = __ldcs(reinterpret_cast<const uint4*>(p)); }
  __device__ __forceinline__ float dot(const float* x, float acc) const {
    const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(x + 4);
    acc = fmaf(__uint_as_float(w.x << 16), a.x, acc);
    acc = fmaf(__uint_as_float(w.x & 0xffff0000u), a.y, acc);
    acc = fmaf(__uint_as_float(w.y << 16), a.z, acc);
    acc = fmaf(__uint_as_float(w.y & 0xffff0000u), a.w, acc);
    acc = fmaf(__uint_as_float(w.z << 16), b.x, acc);
    acc = fmaf(__uint_as_float(w.z & 0xffff0000u), b.y, acc);
    acc = fmaf(__uint_as_float(w.w << 16), b.z, acc);
    return fmaf(__uint_as_float(w.w & 0xffff0000u), b.w, acc);
  }
  __device__ __forceinline__ void unpack(float (&o)[8]) const {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(u[i] << 16);
      o[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
  }
};

// Items 0 .. n - 1 dealt to the threads, U loads of a thread in flight: put(i, load(i)).
template <int U, typename Load, typename Put>
__device__ __forceinline__ void batched(int n, int first, int threads, Load load, Put put) {
  for (int i0 = first; i0 < n; i0 += U * threads) {
    decltype(load(0)) v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * threads < n) v[u] = load(i0 + u * threads);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * threads < n) put(i0 + u * threads, v[u]);
  }
}
struct Pair4 {
  float4 a, b;
};
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float sq4(const float4& a) { return a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w; }

// n / d for n >= 0, d > 0; inv: division_factor(d) from the host. A division by a value that is not known at compile time is
// some 200 cycles of a dependent chain (detatar-0.6b, 1000 + 64 tokens: 99.6 -> 97.0 ms without them). inv d is 2^32 - e with 1 <= e <= d, so the product is short by less than one.
__device__ __forceinline__ int quotient(int n, int d, unsigned inv) {
  const unsigned q = __umulhi(static_cast<unsigned>(n), inv);
  return static_cast<int>(q + (static_cast<unsigned>(n) - q * static_cast<unsigned>(d) >= static_cast<unsigned>(d) ? 1u : 0u));
}

// The same for a divisor that only the device knows, d < 2^24, and a quotient below 2^20: the approximate division's two ulp and the
// roundings of its operands are less than one half there, so the quotient is at most one off.
__device__ __forceinline__ int small_quotient(int x, int d) {
  const int q = static_cast<int>(__fdividef(static_cast<float>(x), static_cast<float>(d))), r = x - q * d;
  return q + (r >= d ? 1 : 0) - (r < 0 ? 1 : 0);
}
__device__ __forceinline__ int quotient(int x, int d) { return x < (1 << 20) ? small_quotient(x, d) : x / d; }

// V neighbouring columns.
template <int V>
struct Cols {
  float v[V];
  __device__ __forceinline__ void load(const float* p) {   // of memory that other CTAs write
    if constexpr (V == 4) {
      const float4 f = ldg4(p);
      v[0] = f.x;
      v[1] = f.y;
      v[2] = f.z;
      v[3] = f.w;
    } else {
      v[0] = ldg_f(p);
    }
  }
  template <typename U>
  __device__ __forceinline__ void get(const U* p) {   // weights, shared memory
    if constexpr (V == 4) {
      const float4 f = load4(p);
      v[0] = f.x;
      v[1] = f.y;
      v[2] = f.z;
      v[3] = f.w;
    } else {
      v[0] = to_f(*p);
    }
  }
  __device__ __forceinline__ void put(float* p) const {
    if constexpr (V == 4) store4(p, make_float4(v[0], v[1], v[2], v[3]));
    else *p = v[0];
  }
};

// A given token may lie outside the vocabulary: its embedding row is zeros, and it is counted in the status word.
__device__ __forceinline__ bool known_id(const TokenArgs& a, int64_t tok) { return tok >= 0 && tok < a.vocab; }

}  // namespace hybrid
}  // namespace ctdk
