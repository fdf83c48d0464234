// Persistent token kernel of the preset decoders (decode_token.cu): one cooperative launch runs one or
// more tokens through all layers.
#pragma once

#include "token_ring.cuh"

namespace ctdk {

constexpr int kTokenMaxLayers = 40;
constexpr int kTokenMaxGrid = 256;
constexpr int kTokenMaxSplits = 32;   // key ranges per kv head of the token attention

struct TokenLayer {
  int64_t w_in, wq, wo, wqn, wkn, w_post, wg, wd;   // offsets into the parameter arena (wqn = -1: no QK-Norm)
};

// A vector that travels between CTAs: one 64-bit word per value, the value in the low half and the number
// of the exchange that wrote it in the high half.
using Word = unsigned long long;

struct TokenKernelArgs {
  const float* P;
  TokenLayer lw[kTokenMaxLayers];
  int64_t embed, norm;
  int L, hid, I, D, H, Hk, group, head_groups, V, QKVN, max_seq;   // group: H / Hk, attended to in head_groups parts
  int qk_norm;
  float eps, scale;
  const float2* table;      // [max_seq][D/2] (cos, sin)
  float *kcache, *vcache;   // [L][Hk][max_seq][D]
  float* logits;
  Word *x, *hm, *qkv, *part, *attn, *act, *best;
  RingRows product[5];         // QKV, O, gate|up, down, head
  int second_at, tile_at, tiles_over, front_floats, residual_floats, stages, stage_bytes;   // shared memory (decode_token.cu): the second place of the vector (0: there is one only), ...
  int tile_bytes;   // of a place for cached keys and values, of which there are two
  int64_t* cur_token;
  int* counters;
  unsigned int* sync;          // [2]: abort flag
  int64_t* out_tokens;         // null: one token, logits only, counters untouched
  int out_offset, n_tokens;
  int* status;
};

// Words of all exchanged vectors of a model.
int64_t token_words(int hid, int QKVN, int I, int H, int D);
// CTAs of the kernel for this model, 0 when it does not take the model.
int token_grid(const TokenKernelArgs& a);
// Clears `words` (token_words() of them) and launches.
int token_launch(TokenKernelArgs& a, Word* words, int grid, cudaStream_t s);

}  // namespace ctdk
