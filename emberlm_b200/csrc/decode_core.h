// What every decoder family shares: the position and token counters in device memory, the logits of
// the last position, and the request loop of decode_api.cu (prefill, portions, single steps, greedy
// bursts). A family (decode.cu: the five presets; hybrid.cu: layer-list models) supplies the forward
// passes and owns its caches and recurrent states.
#pragma once

#include "common.cuh"

namespace ctdk {

struct DecoderBase {
  int vocab = 0, max_seq = 0;
  float* logits = nullptr;        // [vocab], device
  int64_t* cur_token = nullptr;   // device: the token a token pass reads
  int* counters = nullptr;        // device: position, tokens generated, scratch, -, 64-bit argmax word
  cudaGraphExec_t graph = nullptr;
  int64_t* graph_out = nullptr;
  cudaStream_t graph_stream = nullptr;
  // Host mirror of the request: tokens run as portions, tokens the greedy loop emitted, tokens fed by step().
  int64_t prompt_len = 0, generated = 0, stepped = 0;

  virtual ~DecoderBase() {
    if (graph != nullptr) cudaGraphExecDestroy(graph);
  }
  // Runs ids[0, T) (device) at positions pos .. pos + T - 1 on the cache and state the positions before
  // left behind (pos == 0: an empty sequence). n_want >= 0: the logits of the rows want[0, n_want)
  // (host, indices into the portion) go to want_logits [n_want, vocab] (device). n_want < 0: those of
  // the last row go to `logits`. Does not touch the counters.
  virtual int portion(const int64_t* ids, int64_t T, int64_t pos, const int32_t* want, int64_t n_want,
                      float* want_logits, cudaStream_t s) = 0;
  // One token pass: *cur_token at position counters[0] -> logits. Does not touch the counters.
  virtual int token_forward(cudaStream_t s) = 0;
  // n greedy tokens in one launch, appended to out_tokens[generated ..], counters advanced. Returns 1
  // when the family has no such kernel for this model (the caller replays token passes).
  virtual int burst(int64_t n, int64_t* out_tokens, cudaStream_t s) = 0;
};

// First index of the maximum as an atomicMax key: floats ordered as unsigned integers in the high
// half, the smaller index preferred in the low half.
__device__ __forceinline__ unsigned long long argmax_key(float v, int idx) {
  unsigned u = __float_as_uint(v);
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return (static_cast<unsigned long long>(u) << 32) | (0xFFFFFFFFu - static_cast<unsigned>(idx));
}

// Workspace carving in 256-byte steps; base == nullptr only measures.
struct Bump {
  char* base;
  int64_t used = 0;
  explicit Bump(void* b) : base(static_cast<char*>(b)) {}
  void* bytes(int64_t n) {
    void* p = base ? base + used : nullptr;
    used += (n + 255) / 256 * 256;
    return p;
  }
  float* floats(int64_t n) { return static_cast<float*>(bytes(n * 4)); }
};

#define DTRY(expr)                    \
  do {                                \
    int rc_ = (expr);                 \
    if (rc_ != CTDK_OK) return rc_;   \
  } while (0)

#ifdef __CUDACC__
__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
#endif

}  // namespace ctdk
