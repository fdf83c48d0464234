// TF32 GEMM on the 5th-generation tensor cores: C[M,N] = op(A)·op(B) with fp32 operands in
// HBM, fp32 accumulators in tensor memory; and C = A·B^T with bfloat16 operands on the same kernel.
//
// One persistent CTA per SM, 6 warps:
//   warp 0   TMA producer: fills a ring of shared-memory stages (128-byte swizzled tiles),
//            one elected lane, plain (non-multicast) cp.async.bulk.tensor loads.
//   warp 1   MMA issuer: one elected lane issues tcgen05.mma.kind::tf32 (M=128, N=BN, K=8)
//            four times per 32-float stage and releases the stage with tcgen05.commit.
//   warps 2-5 epilogue: read the accumulator with tcgen05.ld (each warp owns one 32-lane
//            quarter of tensor memory) and write C. Two accumulator buffers let the epilogue
//            of tile i overlap the main loop of tile i+1.
// Operands that are contiguous along K are loaded as one box {32 floats, rows}; operands
// contiguous along M or N (the transposed cases of the reference's matmul, emberlm
// src/ops/matmul.cpp:25-47,99-118) are loaded as {32 floats of M/N, 32 rows of K} boxes with
// the 32-byte-atom variant of the 128-byte swizzle and described to the tensor core as
// MN-major. M, N and K tails are zero-filled by TMA bounds
// checking; the epilogue predicates stores. Every mbarrier wait is bounded.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "common.cuh"

namespace ctdk {
namespace {

constexpr int BM = 128;
constexpr int BK = 32;                    // floats per stage along K = one 128-byte swizzle row
constexpr int BKH = 64;                   // the same row in bfloat16
constexpr int kATileBytes = BM * BK * 4;  // 16 KB
constexpr int kChunkBytes = 32 * BK * 4;  // 4 KB: one {32 x 32} box of an MN-major operand
constexpr int kThreads = 192;
constexpr int kGroupM = 16;               // m-blocks per scheduling group (L2 reuse of B tiles)

template <int BN>
struct Cfg {
  static constexpr int kBTileBytes = BN * BK * 4;
  static constexpr int kStageBytes = kATileBytes + kBTileBytes;
  static constexpr int kStages = (BN == 256) ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int kTmemCols = 2 * BN;  // two accumulator buffers
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;
};

struct GemmArgs {
  float* C;
  const float* aux;
  int64_t ldc;
  int M, N, K;
  int epilogue;
  int vec_ok;  // C (and aux) rows are 16-byte aligned and N%4==0
  int splits;  // K is cut into `splits` ranges; >1: partial tiles are added to C with atomics
  int* status;
  // Grouped product (bfloat16 form): m-block i multiplies with the n_pitch rows of B that belong to group
  // tiles[i], and only the first tiles[max_tiles] m-blocks exist. Null: one group.
  const int32_t* tiles = nullptr;
  int max_tiles = 0, n_pitch = 0;
  // bfloat16 outputs (kOutBf16, kOutGlu)
  __nv_bfloat16* out16 = nullptr;
  int up_row = 0;   // kOutGlu: rows of B between a gate row and its up row; N counts pairs
  // lead > 0: the 3xTF32 form A B + A B2 + A2 B. The first `lead` of the `splits` ranges share the first product, the
  // others the two corrections one behind the other.
  int lead = 0;
  // The same form with two runs a unit: range `split` of the first product in one accumulator, range `split` of the
  // corrections in the other, one add of their sum. Up to two units a tile, the order of the adds to a zeroed C does not show.
  int two_runs = 0;
};
// The k-blocks of run `run` of range `split`; those of the corrections count from k_blocks on.
__device__ __forceinline__ void k_range(const GemmArgs& args, int split, int run, int k_blocks, int& kb0, int& kb1) {
  int first = 0, total = k_blocks, part = split, parts = args.splits;
  if (run > 0) {
    first = k_blocks;
    total = 2 * k_blocks;
  } else if (args.lead > 0) {
    if (split < args.lead) {
      parts = args.lead;
    } else {
      first = k_blocks;
      total = 2 * k_blocks;
      part -= args.lead;
      parts -= args.lead;
    }
  }
  kb0 = first + static_cast<int>(static_cast<int64_t>(part) * total / parts);
  kb1 = first + static_cast<int>(static_cast<int64_t>(part + 1) * total / parts);
}

// What the epilogue writes: fp32 sums, the same as bfloat16, or bfloat16 silu(gate) up of the two halves of
// a tile's columns (the first half holds gate rows of B, the second their up rows).
enum GemmOut { kOutF32 = 0, kOutBf16 = 1, kOutGlu = 2 };

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Instruction descriptor: D=F32 (bit 4), A,B format at bits 7 and 10 (kind::tf32: 2 = TF32;
// kind::f16: 1 = BF16), major-ness bits 15/16 (0 = K-major, 1 = MN-major), N>>3 at bit 17, M>>4 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc(bool a_mn, bool b_mn, int n, uint32_t fmt = 2u) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(a_mn) << 15) |
         (static_cast<uint32_t>(b_mn) << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(BM >> 4) << 24);
}

__device__ __forceinline__ void tile_coords(int tile, int m_blocks, int n_blocks, int& mb,
                                            int& nb) {
  const int per_group = kGroupM * n_blocks;
  const int g = tile / per_group;
  const int first_m = g * kGroupM;
  const int gm = min(kGroupM, m_blocks - first_m);
  const int local = tile - g * per_group;
  mb = first_m + local % gm;
  nb = local / gm;
}

// BF16: bfloat16 operands, both K-major. A stage row is 128 bytes either way and an MMA takes 32 of
// them (8 TF32 or 16 bfloat16 values), so tiles, swizzle and descriptors are the same bytes.
//
// Launched as a dependent kernel, but it does not let the next one start early (nor does the cluster kernel below): its grid
// often leaves SMs idle, and a successor's CTAs that arrive while it runs are all placed on those, several to an SM. Prompt
// of 1300 tokens of zutalix-0.6b 6.22 -> 5.92 ms without that, of 90 tokens 3.25 -> 3.01; SmolLM2-135M training on
// 1 x 127 positions 5.03 -> 4.95, on 4 x 511 10.64 -> 10.49.
template <int BN, bool A_MN, bool B_MN, bool BF16, int OUT>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_tf32_kernel(const __grid_constant__ CUtensorMap tmA,
                     const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA2,
                     const __grid_constant__ CUtensorMap tmB2, const GemmArgs args) {
  static_assert(!BF16 || (!A_MN && !B_MN), "bfloat16 operands are K-major");
  static_assert(OUT == kOutF32 || BF16, "bfloat16 outputs go with bfloat16 operands");
  constexpr int TN = OUT == kOutGlu ? BN / 2 : BN;   // output columns of a tile
  using C = Cfg<BN>;
  constexpr int kElems = BF16 ? BKH : BK;   // values of a stage row
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes);
  uint64_t* full = bars;                      // [kStages]
  uint64_t* empty = bars + C::kStages;        // [kStages]
  uint64_t* tfull = bars + 2 * C::kStages;    // [2]
  uint64_t* tempty = tfull + 2;               // [2]
  uint64_t* final_bar = tempty + 2;           // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(final_bar + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 4);
    }
    mbar_init(final_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();     // operands (and C, when it is accumulated into) come from earlier kernels
  const bool grouped = BF16 && args.tiles != nullptr;
  const int m_blocks = grouped ? args.tiles[args.max_tiles] : (args.M + BM - 1) / BM;
  const int n_blocks = (args.N + TN - 1) / TN;
  const int num_tiles = m_blocks * n_blocks;
  const int k_blocks = (args.K + kElems - 1) / kElems;
  const int num_units = num_tiles * args.splits;  // unit u: tile u % num_tiles, k-range u / num_tiles
  const int two = !BF16 && args.two_runs != 0 ? 1 : 0;   // log2 of the runs of a unit

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        const int unit = blockIdx.x + (it >> two) * gridDim.x;
        if (unit >= num_units) break;
        int mb, nb;
        tile_coords(unit % num_tiles, m_blocks, n_blocks, mb, nb);
        const int m0 = mb * BM, n0 = nb * TN;
        const int b_row = grouped ? n0 + args.tiles[mb] * args.n_pitch : n0;
        const int split = unit / num_tiles;
        int kb0, kb1;
        k_range(args, split, it & two, k_blocks, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&empty[s], ph ^ 1u, args.status, 1)) {
            ok = false;
            break;
          }
          unsigned char* a_dst = smem + s * C::kStageBytes;
          unsigned char* b_dst = a_dst + kATileBytes;
          mbar_expect_tx(&full[s], C::kStageBytes);
          const int sweep = kb < k_blocks ? 0 : (kb < 2 * k_blocks ? 1 : 2), k0 = (kb - sweep * k_blocks) * kElems;
          const CUtensorMap* ma = sweep == 2 ? &tmA2 : &tmA;
          const CUtensorMap* mbp = sweep == 1 ? &tmB2 : &tmB;
          if (A_MN) {
#pragma unroll
            for (int c = 0; c < BM / 32; ++c)
              tma_load_2d(a_dst + c * kChunkBytes, ma, &full[s], m0 + 32 * c, k0);
          } else {
            tma_load_2d(a_dst, ma, &full[s], k0, m0);
          }
          if (B_MN) {
#pragma unroll
            for (int c = 0; c < BN / 32; ++c)
              tma_load_2d(b_dst + c * kChunkBytes, mbp, &full[s], n0 + 32 * c, k0);
          } else {
            tma_load_2d(b_dst, mbp, &full[s], k0, b_row);
            if (OUT == kOutGlu) tma_load_2d(b_dst + C::kBTileBytes / 2, mbp, &full[s], k0, b_row + args.up_row);
          }
          if (++s == C::kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(A_MN, B_MN, BN, BF16 ? 1u : 2u);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = 0; ok; ++it) {
        const int unit = blockIdx.x + (it >> two) * gridDim.x;
        if (unit >= num_units) break;
        const int split = unit / num_tiles;
        int kb0, kb1;
        k_range(args, split, it & two, k_blocks, kb0, kb1);
        const int acc = it & 1;
        const uint32_t acc_ph = (static_cast<uint32_t>(it) >> 1) & 1u;
        if (!mbar_wait_bounded(&tempty[acc], acc_ph ^ 1u, args.status, 2)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&full[s], ph, args.status, 3)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
          const uint32_t b_addr = a_addr + kATileBytes;
#pragma unroll
          for (int ks = 0; ks < BK / 8; ++ks) {
            // K-major (SWIZZLE_128B): the 8-float k-slice starts 32 bytes further inside the
            // swizzled row; rows are 128 bytes apart, 8-row groups 1024 bytes apart (SBO).
            // MN-major (SWIZZLE_128B_BASE32B): a k-slice is 8 rows of 128 bytes = two 4-row
            // swizzle groups 512 bytes apart (SBO); the 32-float chunks along M/N are
            // kChunkBytes apart (LBO).
            const uint64_t adesc =
                A_MN ? make_smem_desc(a_addr + ks * 1024, kChunkBytes, 512, kLayoutSw128Base32)
                     : make_smem_desc(a_addr + ks * 32, 16, 1024, kLayoutSw128);
            const uint64_t bdesc =
                B_MN ? make_smem_desc(b_addr + ks * 1024, kChunkBytes, 512, kLayoutSw128Base32)
                     : make_smem_desc(b_addr + ks * 32, 16, 1024, kLayoutSw128);
            if (BF16) umma_bf16(d_tmem, adesc, bdesc, idesc, (kb != kb0 || ks != 0) ? 1u : 0u);
            else umma_tf32(d_tmem, adesc, bdesc, idesc, (kb != kb0 || ks != 0) ? 1u : 0u);
          }
          umma_commit(&empty[s]);  // stage is free once these MMAs have read it
          if (++s == C::kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok) umma_commit(&tfull[acc]);  // accumulator complete
      }
      // All MMAs retired before tensor memory is released.
      umma_commit(final_bar);
      mbar_wait_bounded(final_bar, 0, args.status, 4);
    }
    __syncwarp();
  } else {
    // ------------------------------- epilogue -------------------------------
    const int q = warp & 3;  // tensor-memory lane quarter this warp may access
    const int row_in_tile = q * 32 + lane;
    int it = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x, ++it) {
      int mb, nb;
      tile_coords(unit % num_tiles, m_blocks, n_blocks, mb, nb);
      const bool first_split = unit < num_tiles;
      const bool atomic = args.splits > 1;
      const int acc = two != 0 ? 0 : it & 1;
      const uint32_t acc_ph = (static_cast<uint32_t>(it) >> (1 - two)) & 1u;
      if (!mbar_wait_bounded(&tfull[acc], acc_ph, args.status, 5) || (two != 0 && !mbar_wait_bounded(&tfull[1], acc_ph, args.status, 5))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int64_t grow = static_cast<int64_t>(mb) * BM + row_in_tile;
      const bool row_ok = grow < args.M;
      float* crow = args.C + grow * args.ldc;
      const float* xrow = args.aux != nullptr ? args.aux + grow * args.ldc : nullptr;
      const uint32_t t_row = tmem_base + static_cast<uint32_t>(acc * BN) +
                             (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (OUT != kOutF32) {
        __nv_bfloat16* orow = args.out16 + grow * args.ldc;
#pragma unroll 1
        for (int ch = 0; ch < TN / 32; ++ch) {
          const int col0 = nb * TN + ch * 32;
          if (col0 >= args.N) break;  // warp-uniform
          float v[32];
          tmem_ld_32x32(t_row + static_cast<uint32_t>(ch * 32), v);
          if constexpr (OUT == kOutGlu) {
            float u[32];
            tmem_ld_32x32(t_row + static_cast<uint32_t>(TN + ch * 32), u);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] * __fdividef(1.0f, 1.0f + expf(-v[j])) * u[j];
          }
          if (row_ok) {
            if (args.vec_ok && col0 + 32 <= args.N) {
#pragma unroll
              for (int j = 0; j < 32; j += 8)
                *reinterpret_cast<uint4*>(orow + col0 + j) = make_uint4(pack_bf16(v[j], v[j + 1]), pack_bf16(v[j + 2], v[j + 3]),
                                                                        pack_bf16(v[j + 4], v[j + 5]), pack_bf16(v[j + 6], v[j + 7]));
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < args.N) orow[col0 + j] = __float2bfloat16(v[j]);
            }
          }
          __syncwarp();  // tcgen05.ld is warp-collective: reconverge before the next chunk
        }
      }
#pragma unroll 1
      for (int ch = 0; OUT == kOutF32 && ch < BN / 32; ++ch) {
        const int col0 = nb * BN + ch * 32;
        if (col0 >= args.N) break;  // warp-uniform
        float v[32];
        tmem_ld_32x32(t_row + static_cast<uint32_t>(ch * 32), v);
        if (!BF16 && two != 0) {
          float w[32];
          tmem_ld_32x32(t_row + static_cast<uint32_t>(BN + ch * 32), w);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += w[j];
        }
        if (!row_ok) {
          // rows past M hold zero-filled garbage: nothing to store
        } else if (atomic) {
          // split-K: C was zeroed (STORE / RESIDUAL) or holds the running sum (ACCUMULATE);
          // every k-range adds its partial tile, the first one also adds the residual.
          const bool add_aux = first_split && args.epilogue == CTDK_EPI_RESIDUAL;
          if (args.vec_ok && col0 + 32 <= args.N) {
            float4* c4 = reinterpret_cast<float4*>(crow + col0);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float4 r = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
              if (add_aux) {
                const float4 x = reinterpret_cast<const float4*>(xrow + col0)[j];
                r.x += x.x;
                r.y += x.y;
                r.z += x.z;
                r.w += x.w;
              }
              atomicAdd(&c4[j], r);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int col = col0 + j;
              if (col < args.N) atomicAdd(&crow[col], v[j] + (add_aux ? xrow[col] : 0.0f));
            }
          }
        } else if (args.vec_ok && col0 + 32 <= args.N) {
          float4* c4 = reinterpret_cast<float4*>(crow + col0);
          if (args.epilogue == CTDK_EPI_STORE) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              c4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          } else {
            const float4* x4 = args.epilogue == CTDK_EPI_ACCUMULATE
                                   ? reinterpret_cast<const float4*>(crow + col0)
                                   : reinterpret_cast<const float4*>(xrow + col0);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 x = x4[j];
              c4[j] = make_float4(v[4 * j] + x.x, v[4 * j + 1] + x.y, v[4 * j + 2] + x.z,
                                  v[4 * j + 3] + x.w);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int col = col0 + j;
            if (col < args.N) {
              float r = v[j];
              if (args.epilogue == CTDK_EPI_ACCUMULATE) r += crow[col];
              else if (args.epilogue == CTDK_EPI_RESIDUAL) r += xrow[col];
              crow[col] = r;
            }
          }
        }
        __syncwarp();  // tcgen05.ld is warp-collective: reconverge before the next chunk
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&tempty[acc]);
        if (two != 0) mbar_arrive(&tempty[1]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// ----------------------------------------------------------------------------------------
// K split over a cluster: products with too few tiles for the chip (a few hundred rows)
// ----------------------------------------------------------------------------------------
// A one-CTA tile of 128 x 128 takes about 0.2 us a k-block however idle the rest of the chip is: SmolLM2-135M on 127
// rows has 5 to 24 tiles a product and spent 14 to 15 us on each, three quarters of it in the serial main loop. Here the
// S CTAs of a cluster (2, 4 or 8) share a tile: each multiplies one range of K into its tensor memory, sends every other
// CTA its columns of that partial tile through distributed shared memory, and after one cluster barrier adds up the S
// parts of its own columns in the order of the ranges. Against a split over the grid there is no zeroing launch, no
// atomics, any epilogue, and the result is the same from run to run.
//
// With `sweeps` == 3 the ranges run over three products, A B, A B2 and A2 B: the 3xTF32 form, one launch instead of
// three. Ranges [0, lead) share the first product, the others the two corrections.
template <int BN>
struct ClusterCfg {
  static constexpr int kBTileBytes = BN * BK * 4;
  static constexpr int kStageBytes = kATileBytes + kBTileBytes;
  static constexpr int kStages = BN == 128 ? 4 : 6;
  static constexpr int kPitch = BM + 2;   // float4s between two column groups: rows of a quarter warp in different banks
  static constexpr int kPartBytes = BN / 4 * kPitch * 16;
  static constexpr int kSmemBytes = kStages * kStageBytes + kPartBytes + 1024 /*align*/ + 256 /*barriers*/;
};
struct ClusterArgs {
  float* C;
  const float* aux;
  int64_t ldc;
  int M, N, K, epilogue, vec_ok;
  int S, sweeps, lead;
  int* status;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this CTA's shared memory `addr` in the CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_remote(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int BN, bool A_MN, bool B_MN, bool BF16>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA2,
                        const __grid_constant__ CUtensorMap tmB2, const ClusterArgs args) {
  static_assert(!BF16 || (!A_MN && !B_MN), "bfloat16 operands are K-major");
  using C = ClusterCfg<BN>;
  constexpr int kElems = BF16 ? BKH : BK;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  float4* parts = reinterpret_cast<float4*>(smem + C::kStages * C::kStageBytes);   // [S][columns / 4][kPitch]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes + C::kPartBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::kStages;
  uint64_t* tfull = bars + 2 * C::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  cluster_sync();   // every CTA of the cluster is there before its shared memory is written
  pdl_wait();

  const int S = args.S, rank = static_cast<int>(blockIdx.x) % S;
  const int m_blocks = (args.M + BM - 1) / BM, n_blocks = (args.N + BN - 1) / BN;
  const int k_blocks = (args.K + kElems - 1) / kElems;
  // this CTA's range of the sweeps' k-blocks
  int kb0, kb1;
  if (args.sweeps == 1) {
    kb0 = rank * k_blocks / S;
    kb1 = (rank + 1) * k_blocks / S;
  } else if (rank < args.lead) {
    kb0 = rank * k_blocks / args.lead;
    kb1 = (rank + 1) * k_blocks / args.lead;
  } else {
    const int n = S - args.lead, r = rank - args.lead;
    kb0 = k_blocks + r * 2 * k_blocks / n;
    kb1 = k_blocks + (r + 1) * 2 * k_blocks / n;
  }
  const int cols = BN / S, quads = cols / 4;   // columns of the tile that this CTA finishes
  int s = 0;
  uint32_t ph = 0;
  bool ok = true;
  int mb, nb;
  tile_coords(static_cast<int>(blockIdx.x) / S, m_blocks, n_blocks, mb, nb);
  if (warp == 0) {
    if (lane == 0) {
      const int m0 = mb * BM, n0 = nb * BN;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (!mbar_wait_bounded(&empty[s], ph ^ 1u, args.status, 1)) {
          ok = false;
          break;
        }
        unsigned char* a_dst = smem + s * C::kStageBytes;
        unsigned char* b_dst = a_dst + kATileBytes;
        mbar_expect_tx(&full[s], C::kStageBytes);
        const int sweep = kb / k_blocks, k0 = (kb - sweep * k_blocks) * kElems;
        const CUtensorMap* ma = sweep == 2 ? &tmA2 : &tmA;
        const CUtensorMap* mbp = sweep == 1 ? &tmB2 : &tmB;
        if (A_MN) {
#pragma unroll
          for (int c = 0; c < BM / 32; ++c) tma_load_2d(a_dst + c * kChunkBytes, ma, &full[s], m0 + 32 * c, k0);
        } else {
          tma_load_2d(a_dst, ma, &full[s], k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int c = 0; c < BN / 32; ++c) tma_load_2d(b_dst + c * kChunkBytes, mbp, &full[s], n0 + 32 * c, k0);
        } else {
          tma_load_2d(b_dst, mbp, &full[s], k0, n0);
        }
        if (++s == C::kStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(A_MN, B_MN, BN, BF16 ? 1u : 2u);
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (!mbar_wait_bounded(&full[s], ph, args.status, 3)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes), b_addr = a_addr + kATileBytes;
#pragma unroll
        for (int ks = 0; ks < BK / 8; ++ks) {   // descriptors as in gemm_tf32_kernel
          const uint64_t adesc = A_MN ? make_smem_desc(a_addr + ks * 1024, kChunkBytes, 512, kLayoutSw128Base32)
                                      : make_smem_desc(a_addr + ks * 32, 16, 1024, kLayoutSw128);
          const uint64_t bdesc = B_MN ? make_smem_desc(b_addr + ks * 1024, kChunkBytes, 512, kLayoutSw128Base32)
                                      : make_smem_desc(b_addr + ks * 32, 16, 1024, kLayoutSw128);
          if (BF16) umma_bf16(tmem_base, adesc, bdesc, idesc, (kb != kb0 || ks != 0) ? 1u : 0u);
          else umma_tf32(tmem_base, adesc, bdesc, idesc, (kb != kb0 || ks != 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        if (++s == C::kStages) {
          s = 0;
          ph ^= 1u;
        }
      }
      umma_commit(tfull);   // also behind a wait that ran out: nothing of this CTA is then in flight when it goes on
      mbar_wait_bounded(tfull, 0, args.status, 4);
    }
    __syncwarp();
  } else {
    const int q = warp & 3, row = q * 32 + lane;
    if (!mbar_wait_bounded(tfull, 0, args.status, 5)) ok = false;
    tc_fence_after();
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
    for (int ch = 0; ch < BN / 32; ++ch) {
      float v[32];
      tmem_ld_32x32(t_row + static_cast<uint32_t>(ch * 32), v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int col = ch * 32 + 4 * j, dst = col / cols, quad = (col - dst * cols) >> 2;
        store_remote(in_cta(smem_u32(parts + (rank * quads + quad) * C::kPitch + row), static_cast<uint32_t>(dst)), v[4 * j], v[4 * j + 1],
                     v[4 * j + 2], v[4 * j + 3]);
      }
      __syncwarp();
    }
    tc_fence_before();
  }
  __syncwarp();
  // all parts of this CTA's columns are there, and its tensor memory has been read; nothing reaches another CTA's memory
  // from here on, so each may leave
  cluster_sync();
  tc_fence_after();
  for (int i = threadIdx.x; i < quads * BM; i += kThreads) {
    const int quad = i % quads, row = i / quads;
    float4 v = parts[quad * C::kPitch + row];
    for (int r = 1; r < S; ++r) {
      const float4 w = parts[(r * quads + quad) * C::kPitch + row];
      v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
    }
    const int64_t grow = static_cast<int64_t>(mb) * BM + row;
    const int col = nb * BN + rank * cols + 4 * quad;
    if (grow >= args.M || col >= args.N) continue;
    float* c = args.C + grow * args.ldc + col;
    const float* x = args.epilogue == CTDK_EPI_ACCUMULATE ? c : (args.epilogue == CTDK_EPI_RESIDUAL ? args.aux + grow * args.ldc + col : nullptr);
    if (args.vec_ok && col + 4 <= args.N) {
      if (x != nullptr) {
        const float4 w = *reinterpret_cast<const float4*>(x);
        v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
      }
      *reinterpret_cast<float4*>(c) = v;
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (col + k < args.N) c[k] = e[k] + (x != nullptr ? x[k] : 0.0f);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

// ----------------------------------------------------------------------------------------
// Host side
// ----------------------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  return g_encode;
}

bool tma_rounds_to_tf32() {
  // CTDK_TMA_F32=1 loads raw fp32 bits (the tensor core then ignores the low mantissa bits);
  // the default asks the copy engine for the TF32 data type.
  static const bool raw = [] {
    const char* e = std::getenv("CTDK_TMA_F32");
    return e != nullptr && e[0] == '1';
  }();
  return !raw;
}

// 2-D map over a row-major fp32 matrix: dim0 = contiguous extent `inner`, dim1 = `outer`
// rows `ld` floats apart; box = {32, box_rows}; 128-byte rows swizzled in 16-byte chunks
// (K-major tiles) or 32-byte chunks (MN-major tiles); out-of-range reads give 0.
int make_map(CUtensorMap* map, const float* base, int64_t inner, int64_t outer, int64_t ld,
             int box_rows, bool mn_major, bool exact_fp32) {
  auto enc = encode_fn();
  if (enc == nullptr) return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * sizeof(float)};
  cuuint32_t box[2] = {32u, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1u, 1u};
  const CUtensorMapDataType dt = (!exact_fp32 && tma_rounds_to_tf32())
                                     ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32
                                     : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = enc(map, dt, 2, const_cast<float*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled failed (%d): inner=%lld outer=%lld ld=%lld",
                static_cast<int>(r), static_cast<long long>(inner),
                static_cast<long long>(outer), static_cast<long long>(ld));
  return CTDK_OK;
}

}  // namespace

int encode_tensor_map(CUtensorMap* map, const float* base, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box, bool atom32) {
  auto enc = encode_fn();
  if (enc == nullptr) return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t d[5], st[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i + 1 < rank) st[i] = strides_bytes[i];
  }
  const CUtensorMapDataType dt =
      tma_rounds_to_tf32() ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = enc(map, dt, rank, const_cast<float*>(base), d, st, bx, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   atom32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled failed (%d), rank %d", static_cast<int>(r), rank);
  return CTDK_OK;
}

namespace {

template <int BN, bool A_MN, bool B_MN, bool BF16 = false, int OUT = kOutF32>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args,
           cudaStream_t stream, const CUtensorMap* ta2 = nullptr, const CUtensorMap* tb2 = nullptr) {
  using C = Cfg<BN>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  auto* kern = gemm_tf32_kernel<BN, A_MN, B_MN, BF16, OUT>;
  constexpr int TN = OUT == kOutGlu ? BN / 2 : BN;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess)
      return fail(CTDK_ELAUNCH, "gemm: cannot opt in to %d bytes of shared memory: %s",
                  C::kSmemBytes, cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  const int m_blocks = args.tiles != nullptr ? args.max_tiles : (args.M + BM - 1) / BM, n_blocks = (args.N + TN - 1) / TN;
  const int tiles = m_blocks * n_blocks * args.splits;
  const int sms = sm_count();
  const int grid = tiles < sms ? tiles : sms;
  const cudaError_t le = launch_pdl(kern, dim3(grid), dim3(kThreads), C::kSmemBytes, stream, ta, tb, ta2 != nullptr ? *ta2 : ta,
                                    tb2 != nullptr ? *tb2 : tb, args);
  if (le != cudaSuccess) return fail(CTDK_ELAUNCH, "gemm: launch failed: %s", cudaGetErrorString(le));
  return check_launch("ctdk_gemm(tcgen05)");
}

template <int BN>
int dispatch_major(bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb,
                   const GemmArgs& args, cudaStream_t stream, const CUtensorMap* ta2 = nullptr, const CUtensorMap* tb2 = nullptr) {
  if (!a_mn && !b_mn) return launch<BN, false, false>(ta, tb, args, stream, ta2, tb2);
  if (!a_mn && b_mn) return launch<BN, false, true>(ta, tb, args, stream, ta2, tb2);
  if (a_mn && !b_mn) return launch<BN, true, false>(ta, tb, args, stream, ta2, tb2);
  return launch<BN, true, true>(ta, tb, args, stream, ta2, tb2);
}

template <int BN, bool A_MN, bool B_MN, bool BF16 = false>
int launch_cluster(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& ta2, const CUtensorMap& tb2, const ClusterArgs& args,
                   cudaStream_t stream) {
  using C = ClusterCfg<BN>;
  auto* kern = gemm_cluster_kernel<BN, A_MN, B_MN, BF16>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return fail(CTDK_ELAUNCH, "gemm(cluster): shared memory opt-in failed: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  const int tiles = ((args.M + BM - 1) / BM) * ((args.N + BN - 1) / BN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * args.S);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = args.S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tb, ta2, tb2, args);
  if (e != cudaSuccess) return fail(CTDK_ELAUNCH, "gemm(cluster): launch failed: %s", cudaGetErrorString(e));
  return check_launch("ctdk_gemm(tcgen05, cluster)");
}
template <int BN>
int launch_cluster_major(bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& ta2, const CUtensorMap& tb2,
                         const ClusterArgs& args, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_cluster<BN, false, false>(ta, tb, ta2, tb2, args, stream);
  if (!a_mn && b_mn) return launch_cluster<BN, false, true>(ta, tb, ta2, tb2, args, stream);
  if (a_mn && !b_mn) return launch_cluster<BN, true, false>(ta, tb, ta2, tb2, args, stream);
  return launch_cluster<BN, true, true>(ta, tb, ta2, tb2, args, stream);
}

// Clusters of S CTAs (one per SM) that run at a time, 0 when that cannot be told. A GPC's SMs that do not fill a cluster
// stay idle, and how many these are differs from card to card: 74, 33 and 15 clusters of 2, 4 and 8 here. One tile more than
// that is a second wave: 16 tiles on clusters of 8 took 20.3 us where 15 would take 12.5 and the plain kernel 12.1
// (64 x 1024 x 4096).
int clusters_of(int S) {
  static std::mutex mu;
  static int most[64][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lk(mu);
  if (most[dev][S] == 0) {
    auto* kern = gemm_cluster_kernel<128, false, false, false>;
    constexpr int smem = ClusterCfg<128>::kSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    most[dev][S] = n;
  }
  return std::min(most[dev][S], sm_budget() / S);
}

// Estimated time of a product on the cluster kernel in microseconds, and its tile width and cluster size. Fitted to
// dependent launches of 84 products (16 to 255 rows, 576 to 16384 columns and terms; bfloat16 the same within 15 %): a
// k-block of a range takes 0.31 us at 64 columns and 0.36 at 128, all else 5.6 and 8.0.
double choose_cluster(int64_t M, int64_t N, int64_t k_blocks, int* bn_out, int* s_out) {
  double best = 1e300;
  const int widths[2] = {128, 64}, most[9] = {0, 0, clusters_of(2), 0, clusters_of(4), 0, 0, 0, clusters_of(8)};
  for (int w : widths) {
    const int64_t tiles = ((M + BM - 1) / BM) * ((N + w - 1) / w);
    for (int S = 8; S >= 2; S /= 2) {
      if (k_blocks < 2 * S) continue;   // every CTA has a range worth its share of the exchange
      if (tiles > most[S]) continue;   // a second wave of clusters would double the time
      const double t = static_cast<double>((k_blocks + S - 1) / S) * (w == 128 ? 0.36 : 0.31) + (w == 128 ? 8.0 : 5.6);
      if (t < best * 0.97) {
        best = t;
        *bn_out = w;
        *s_out = S;
      }
    }
  }
  return best;
}

}  // namespace

int gemm_tcgen05_2cta(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, bool a_mn, bool b_mn,
                      bool a3d, bool b3d, int tma_out, float* C, const float* aux, int64_t ldc, int M, int N, int K,
                      int epilogue, int vec_ok, int splits, int* status, cudaStream_t stream);

int gemm_tcgen05_2cta_swiglu(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tgu, const CUtensorMap& tact,
                             int M, int N, int K, int* status, cudaStream_t stream);

// gu[M, 2I] = A[M, K] W[2I, K]^T and act[M, I] = silu(gu[:, :I]) * gu[:, I:] in one paired-CTA launch.
// Returns CTDK_OK after enqueueing, a negative status, or 1 when the shape is not eligible.
int gemm_swiglu_tcgen05(const float* A, const float* W, float* gu, float* act, int64_t M, int64_t I, int64_t K,
                        cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(A) || !a16(W) || !a16(gu) || !a16(act) || (K & 3) || (I % 128) != 0) return 1;
  if (M < 256 || M > INT32_MAX || 2 * I > INT32_MAX || K > INT32_MAX || K < 1) return 1;
  CUtensorMap ta, tb, tgu, tact;
  int rc = make_map(&ta, A, K, M, K, BM, false, false);
  if (rc == CTDK_OK) rc = make_map(&tb, W, K, 2 * I, K, 128, false, false);
  if (rc == CTDK_OK) rc = make_map(&tgu, gu, 2 * I, M, 2 * I, 32, false, true);
  if (rc == CTDK_OK) rc = make_map(&tact, act, I, M, I, 32, false, true);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  return gemm_tcgen05_2cta_swiglu(ta, tb, tgu, tact, static_cast<int>(M), static_cast<int>(I), static_cast<int>(K), st, stream);
}

int gemm_tcgen05_2cta_swiglu_bwd(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tgu, const CUtensorMap& tdgu,
                                 bool b3d, int M, int N, int K, int* status, cudaStream_t stream);

// dgu[M, 2I] = SwiGLU backward of (dy[M, K] * Wd[K, I]) against gu[M, 2I], in one paired-CTA launch.
// Returns CTDK_OK after enqueueing, a negative status, or 1 when the shape is not eligible.
int gemm_swiglu_bwd_tcgen05(const float* dy, const float* Wd, const float* gu, float* dgu, int64_t M, int64_t I, int64_t K,
                            cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(dy) || !a16(Wd) || !a16(gu) || !a16(dgu) || (K & 3) || (I % 32) != 0) return 1;
  if (M < 256 || I < 256 || M > INT32_MAX || 2 * I > INT32_MAX || K > INT32_MAX || K < 1) return 1;
  CUtensorMap ta, tb, tgu, tdgu;
  int rc = make_map(&ta, dy, K, M, K, BM, false, false);
  if (rc == CTDK_OK) {
    const uint64_t dims[3] = {32u, static_cast<uint64_t>(K), static_cast<uint64_t>(I / 32)};
    const uint64_t strides[2] = {static_cast<uint64_t>(I) * sizeof(float), 128u};
    const uint32_t box[3] = {32u, 32u, 4u};
    rc = encode_tensor_map(&tb, Wd, 3, dims, strides, box, true);
  }
  if (rc == CTDK_OK) rc = make_map(&tgu, gu, 2 * I, M, 2 * I, 32, false, true);
  if (rc == CTDK_OK) rc = make_map(&tdgu, dgu, 2 * I, M, 2 * I, 32, false, true);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  return gemm_tcgen05_2cta_swiglu_bwd(ta, tb, tgu, tdgu, true, static_cast<int>(M), static_cast<int>(I), static_cast<int>(K), st,
                                      stream);
}

int gemm_tcgen05_2cta_dattn_delta(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& to,
                                  bool b3d, float* delta, int M, int N, int K, int T, int H, int D, int* status,
                                  cudaStream_t stream);

// dattn[M, H*D] = dy[M, K] * Wo[K, H*D] and delta[b, h, t] = sum_d dattn * out over each head, in one paired-CTA
// launch (M = B * T rows). Returns CTDK_OK after enqueueing, a negative status, or 1 when not eligible.
int gemm_dattn_delta_tcgen05(const float* dy, const float* Wo, const float* out, float* dattn, float* delta, int64_t M,
                             int64_t T, int H, int D, int64_t K, cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const int64_t N = static_cast<int64_t>(H) * D;
  if (!a16(dy) || !a16(Wo) || !a16(out) || !a16(dattn) || (K & 3) || (D != 64 && D != 128)) return 1;
  if (M < 256 || N < 256 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX || K < 1 || T < 1 || M % T != 0) return 1;
  CUtensorMap ta, tb, tc, to;
  int rc = make_map(&ta, dy, K, M, K, BM, false, false);
  if (rc == CTDK_OK) {
    const uint64_t dims[3] = {32u, static_cast<uint64_t>(K), static_cast<uint64_t>(N / 32)};
    const uint64_t strides[2] = {static_cast<uint64_t>(N) * sizeof(float), 128u};
    const uint32_t box[3] = {32u, 32u, 4u};
    rc = encode_tensor_map(&tb, Wo, 3, dims, strides, box, true);
  }
  if (rc == CTDK_OK) rc = make_map(&tc, dattn, N, M, N, 32, false, true);
  if (rc == CTDK_OK) rc = make_map(&to, out, N, M, N, 32, false, true);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  return gemm_tcgen05_2cta_dattn_delta(ta, tb, tc, to, true, delta, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                                       static_cast<int>(T), H, D, st, stream);
}

// Upper bound on the k-blocks one unit accumulates in tensor memory (0 = none), per host thread.
// The tensor core's fp32 accumulation loses low bits with every addition, so the error of a product
// grows with the length of the accumulation (measured: 2.1e-5 of the largest element at K = 8192 in
// one run against 1.3e-6 when the same K is added up from 512-deep pieces in fp32). The 3xTF32 mode
// sets it for its leading (hi x hi) product: K is then cut into ranges of at most that many
// k-blocks whose partial tiles are added at L2 in fp32.
static thread_local int t_kblock_limit = 0;
void gemm_set_kblock_limit(int k_blocks) { t_kblock_limit = k_blocks; }

namespace {

// Tile width, K split and one-CTA / paired-CTA kernel for an M x N product of k_blocks stage rows; returns the estimate of
// the one-CTA kernel (k-blocks of a 256-wide tile).
double choose_tile(int64_t M, int64_t N, int64_t k_blocks, int* bn_out, int* splits_out, bool* pair_out) {
  // Tile width and K split: estimated time = rounds of the persistent grid x k-blocks per
  // unit x relative cost of a k-block (a 128-wide tile does half the work of a 256-wide one
  // but moves 2/3 of the operand bytes, hence the 0.6). Splitting K only pays when the output
  // tiles alone cannot fill the SMs (weight gradients: few tiles, K = all tokens).
  const int sms = sm_budget();
  const int64_t m_blocks = (M + BM - 1) / BM;
  int bn = 64, splits = 1;
  double best = static_cast<double>((m_blocks + sms - 1) / sms) * (static_cast<double>(k_blocks) + 6.0) * 0.45;
  if (N > 64) {
    best = 1e300;
    const int widths[2] = {256, 128};
    for (int wi = 0; wi < 2; ++wi) {
      const int w = widths[wi];
      if (w == 256 && N <= 128) continue;
      const int64_t tiles = m_blocks * ((N + w - 1) / w);
      const int max_splits = static_cast<int>(k_blocks / 16 < 1 ? 1 : (k_blocks / 16 > 32 ? 32 : k_blocks / 16));
      for (int sp = 1; sp <= max_splits; ++sp) {
        if (sp > 1 && tiles >= 2 * sms) break;
        const int64_t units = tiles * sp;
        const double rounds = static_cast<double>((units + sms - 1) / sms);
        const double kb = static_cast<double>((k_blocks + sp - 1) / sp);
        // + a fixed per-unit cost (epilogue / atomics) in k-block equivalents
        const double t = rounds * (kb + (sp > 1 ? 12.0 : 6.0)) * (w == 256 ? 1.0 : 0.6);
        if (t < best * 0.97) {
          best = t;
          bn = w;
          splits = sp;
        }
      }
    }
  }

  // Paired-CTA kernel (256 x 256 tile per CTA pair, half of B per CTA): same cost model, a pair
  // round does the work of two 256-wide rounds in about 1.7x the time of one.
  static const bool pair_off = [] {
    const char* e = std::getenv("CTDK_GEMM_1CTA");
    return e != nullptr && e[0] == '1';
  }();
  bool use_pair = false;
  if (!pair_off && M >= 256 && N >= 256) {
    double best1 = 1e300;
    {
      const int64_t tiles = m_blocks * ((N + bn - 1) / bn);
      const double rounds = static_cast<double>((tiles * splits + sms - 1) / sms);
      best1 = rounds * (static_cast<double>((k_blocks + splits - 1) / splits) + (splits > 1 ? 12.0 : 6.0)) *
              (bn == 256 ? 1.0 : (bn == 128 ? 0.6 : 0.4));
    }
    const int pairs = sms / 2;
    const int64_t tiles2 = ((M + 255) / 256) * ((N + 255) / 256);
    const int max_splits = static_cast<int>(k_blocks / 16 < 1 ? 1 : (k_blocks / 16 > 32 ? 32 : k_blocks / 16));
    double bestp = 1e300;
    int sp_best = 1;
    for (int sp = 1; sp <= max_splits; ++sp) {
      if (sp > 1 && tiles2 >= 2 * pairs) break;
      const double rounds = static_cast<double>((tiles2 * sp + pairs - 1) / pairs);
      const double t = rounds * (static_cast<double>((k_blocks + sp - 1) / sp) + (sp > 1 ? 12.0 : 6.0)) * 1.7;
      if (t < bestp * 0.97) {
        bestp = t;
        sp_best = sp;
      }
    }
    // compare per-SM-round costs: a one-CTA round covers `sms` tiles, a pair round `pairs` tiles
    if (bestp < best1 * 2.0 * 0.98) {
      use_pair = true;
      splits = sp_best;
      bn = 256;
    }
  }
  *bn_out = bn;
  *splits_out = splits;
  *pair_out = use_pair;
  return best;
}

// The same estimate in microseconds, of the same measurements as choose_cluster: 0.39 us a unit of choose_tile and 5.9 us
// (bfloat16: 4.0) for all else. A split K also needs the launch that zeroes the output, which takes part in no dependent
// launch, and adds every range's tile at L2: 5 us and 0.2 a range in a training step (1 us between equal products).
double plain_us(double units, int splits, bool bf16) { return 0.39 * units + (bf16 ? 4.0 : 5.9) + (splits > 1 ? 5.0 + 0.2 * splits : 0.0); }

}  // namespace

// Zeroes in front of a product whose ranges of K add to C. Weight gradients (A transposed) run beside the chain of the backward pass,
// where a product that starts earlier takes the SMs of the chain's next kernel: a memset node, behind which it starts later
// (SmolLM2-135M, 64 x 63 positions, 30 gate|up gradients a step: 12.97 -> 12.65 ms; 4 x 511 unchanged). Elsewhere the product is a
// link of the chain: the kernel that overlaps it (SmolLM2-360M, 2 x 700 positions, 97 a step: 14.57 ms, 14.92 with memset nodes).
static int zero_result(float* C, int64_t M, int64_t N, int64_t ldc, bool gradient, cudaStream_t s) {
  if (!gradient) return zero_rows(C, M, N, ldc, s);
  const cudaError_t e = cudaMemset2DAsync(C, static_cast<size_t>(ldc) * sizeof(float), 0, static_cast<size_t>(N) * sizeof(float), static_cast<size_t>(M), s);
  return e == cudaSuccess ? CTDK_OK : fail(CTDK_ELAUNCH, "gemm: memset failed: %s", cudaGetErrorString(e));
}

// Returns CTDK_OK after enqueueing, or 1 when the shape/alignment is not eligible for the
// tensor-core path (the caller then uses the SIMT kernel).
int gemm_tcgen05(const float* A, const float* B, float* Cp, int64_t M, int64_t N, int64_t K,
                 int64_t lda, int64_t ldb, int64_t ldc, int transa, int transb, int epilogue,
                 const float* aux, cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(A) || !a16(B) || (lda & 3) || (ldb & 3)) return 1;
  if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return 1;
  if (M < 1 || N < 8 || K < 1) return 1;

  const bool a_mn = transa != 0;  // A stored [K,M]: contiguous along M
  const bool b_mn = transb == 0;  // B stored [K,N]: contiguous along N
  const int64_t k_blocks = (K + BK - 1) / BK;
  int bn, splits;
  bool use_pair;
  const double units = choose_tile(M, N, k_blocks, &bn, &splits, &use_pair);
  // From 256 rows on the order of additions stays as it is: the forms with a fused epilogue, which begin there, give the
  // same bits as the product and the kernel behind it. (Weight gradients that are split over the grid were tried on
  // clusters: SmolLM2-135M on 4 x 511 positions 10.9 -> 11.4 ms, the clusters hold SMs that the main stream needs.)
  if (!use_pair && t_kblock_limit == 0 && M < 256) {
    int cbn = 0, S = 0;
    if (choose_cluster(M, N, k_blocks, &cbn, &S) < plain_us(units, splits, false)) {
      CUtensorMap ta, tb;
      int rc = a_mn ? make_map(&ta, A, M, K, lda, BK, true, false) : make_map(&ta, A, K, M, lda, BM, false, false);
      if (rc == CTDK_OK) rc = b_mn ? make_map(&tb, B, N, K, ldb, BK, true, false) : make_map(&tb, B, K, N, ldb, cbn, false, false);
      if (rc != CTDK_OK) return rc;
      ClusterArgs c{Cp, aux, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), epilogue, 0, S, 1, 0, device_status_word()};
      c.vec_ok = a16(Cp) && (ldc & 3) == 0 && (aux == nullptr || a16(aux)) ? 1 : 0;
      if (c.status == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
      return cbn == 128 ? launch_cluster_major<128>(a_mn, b_mn, ta, tb, ta, tb, c, stream)
                        : launch_cluster_major<64>(a_mn, b_mn, ta, tb, ta, tb, c, stream);
    }
  }

  if (t_kblock_limit > 0) {
    int64_t need = (k_blocks + t_kblock_limit - 1) / t_kblock_limit;
    if (need > 64) need = 64;
    if (need > splits) splits = static_cast<int>(need);
  }

  CUtensorMap ta, tb;
  int rc;
  // The pair kernel takes an MN-major operand whose contiguous extent is a multiple of 32 through
  // a 3-D map {32 columns, K rows, extent / 32 column groups}: one {32, 32, 4} box per k-block
  // instead of four {32, 32} boxes (issuing a TMA copy costs the producer thread ~140 cycles).
  auto make_map3 = [&](CUtensorMap* m, const float* base, int64_t extent, int64_t ld) {
    const uint64_t dims[3] = {32u, static_cast<uint64_t>(K), static_cast<uint64_t>(extent / 32)};
    const uint64_t strides[2] = {static_cast<uint64_t>(ld) * sizeof(float), 128u};
    const uint32_t box[3] = {32u, 32u, 4u};
    return encode_tensor_map(m, base, 3, dims, strides, box, true);
  };
  const bool a3d = use_pair && a_mn && (M % 32 == 0);
  const bool b3d = use_pair && b_mn && (N % 32 == 0);
  if (a3d) rc = make_map3(&ta, A, M, lda);
  else if (a_mn) rc = make_map(&ta, A, M, K, lda, BK, true, false);
  else rc = make_map(&ta, A, K, M, lda, BM, false, false);
  if (rc != CTDK_OK) return rc;
  if (b3d) rc = make_map3(&tb, B, N, ldb);
  else if (b_mn) rc = make_map(&tb, B, N, K, ldb, BK, true, false);
  else rc = make_map(&tb, B, K, N, ldb, use_pair ? 128 : bn, false, false);
  if (rc != CTDK_OK) return rc;

  if (use_pair) {
    int* st = device_status_word();
    if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
    const int vec = (a16(Cp) && (ldc & 3) == 0 && (aux == nullptr || a16(aux))) ? 1 : 0;
    if (splits > 1 && epilogue != CTDK_EPI_ACCUMULATE) {
      rc = zero_result(Cp, M, N, ldc, transa != 0, stream);
      if (rc != CTDK_OK) return rc;
    }
    // Output through TMA (coalesced, off the load/store pipe): plain store, or an fp32 add at L2
    // for accumulation and for split-K partial tiles. The residual epilogue reads a second
    // matrix and keeps the direct path.
    int tma_out = 0;
    CUtensorMap tc = ta;
    if (vec && epilogue != CTDK_EPI_RESIDUAL) {
      tma_out = (epilogue == CTDK_EPI_ACCUMULATE || splits > 1) ? 2 : 1;
      rc = make_map(&tc, Cp, N, M, ldc, 32, false, true);
      if (rc != CTDK_OK) return rc;
    }
    return gemm_tcgen05_2cta(ta, tb, tc, a_mn, b_mn, a3d, b3d, tma_out, Cp, aux, ldc, static_cast<int>(M),
                             static_cast<int>(N), static_cast<int>(K), epilogue, vec, splits, st, stream);
  }

  GemmArgs args;
  args.C = Cp;
  args.aux = aux;
  args.ldc = ldc;
  args.M = static_cast<int>(M);
  args.N = static_cast<int>(N);
  args.K = static_cast<int>(K);
  args.epilogue = epilogue;
  args.vec_ok = (a16(Cp) && (ldc & 3) == 0 && (aux == nullptr || a16(aux))) ? 1 : 0;
  args.splits = splits;
  args.status = device_status_word();
  if (args.status == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  if (splits > 1 && epilogue != CTDK_EPI_ACCUMULATE) {
    rc = zero_result(Cp, M, N, ldc, transa != 0, stream);
    if (rc != CTDK_OK) return rc;
  }

  switch (bn) {
    case 64: return dispatch_major<64>(a_mn, b_mn, ta, tb, args, stream);
    case 128: return dispatch_major<128>(a_mn, b_mn, ta, tb, args, stream);
    default: return dispatch_major<256>(a_mn, b_mn, ta, tb, args, stream);
  }
}

int encode_tensor_map_bf16(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                           const uint32_t* box) {
  auto enc = encode_fn();
  if (enc == nullptr) return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t d[5], st[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1u;
    if (i + 1 < rank) st[i] = strides_bytes[i];
  }
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, static_cast<cuuint32_t>(rank), const_cast<void*>(base), d, st, bx, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(CTDK_ELAUNCH, "cuTensorMapEncodeTiled failed (%d) for a bfloat16 operand", static_cast<int>(r));
  return CTDK_OK;
}

int gemm_tcgen05_2cta_bf16(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, int tma_out, float* C,
                           int64_t ldc, int M, int N, int K, int vec_ok, int splits, int* status, cudaStream_t stream);

// C[M, N] (fp32) = A[M, K] B[N, K]^T with bfloat16 operands in memory, fp32 accumulation. Pointers
// 16-byte aligned, lda and ldb multiples of 8.
int gemm_bf16_tcgen05(const void* A, const void* B, float* Cp, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb,
                      int64_t ldc, cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  CTDK_REQUIRE(a16(A) && a16(B) && (lda & 7) == 0 && (ldb & 7) == 0, "gemm_bf16: operands must be 16-byte aligned");
  CTDK_REQUIRE(M >= 1 && N >= 8 && K >= 1 && M <= INT32_MAX && N <= INT32_MAX && K <= INT32_MAX, "gemm_bf16: bad shape");
  const int64_t k_blocks = (K + BKH - 1) / BKH;
  int bn, splits;
  bool use_pair;
  const double units = choose_tile(M, N, k_blocks, &bn, &splits, &use_pair);
  int cbn = 0, S = 0;
  const bool cluster = !use_pair && choose_cluster(M, N, k_blocks, &cbn, &S) < plain_us(units, splits, true);
  if (cluster) bn = cbn;
  if (!cluster && bn == 64 && splits == 1)   // one narrow column of tiles (low-rank factors): split K while SMs are idle
    while ((M + BM - 1) / BM * splits * 2 <= sm_budget() && k_blocks / (splits * 2) >= 8) splits *= 2;
  auto map_bf16 = [](CUtensorMap* map, const void* base, int64_t inner, int64_t outer, int64_t ld, int box_rows) {
    const uint64_t dims[2] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer)}, strides[1] = {static_cast<uint64_t>(ld) * 2};
    const uint32_t box[2] = {static_cast<uint32_t>(BKH), static_cast<uint32_t>(box_rows)};
    return encode_tensor_map_bf16(map, base, 2, dims, strides, box);
  };
  CUtensorMap ta, tb;
  int rc = map_bf16(&ta, A, K, M, lda, BM);
  if (rc == CTDK_OK) rc = map_bf16(&tb, B, K, N, ldb, use_pair ? 128 : bn);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  const int vec = (a16(Cp) && (ldc & 3) == 0) ? 1 : 0;
  if (cluster) {
    const ClusterArgs c{Cp, nullptr, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), CTDK_EPI_STORE, vec, S, 1, 0, st};
    return bn == 128 ? launch_cluster<128, false, false, true>(ta, tb, ta, tb, c, stream)
                     : launch_cluster<64, false, false, true>(ta, tb, ta, tb, c, stream);
  }
  if (splits > 1) {
    rc = zero_rows(Cp, M, N, ldc, stream);
    if (rc != CTDK_OK) return rc;
  }
  if (use_pair) {
    int tma_out = 0;
    CUtensorMap tc = ta;
    if (vec) {
      tma_out = splits > 1 ? 2 : 1;
      rc = make_map(&tc, Cp, N, M, ldc, 32, false, true);
      if (rc != CTDK_OK) return rc;
    }
    return gemm_tcgen05_2cta_bf16(ta, tb, tc, tma_out, Cp, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), vec,
                                  splits, st, stream);
  }
  const GemmArgs args{Cp, nullptr, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), CTDK_EPI_STORE, vec, splits, st};
  switch (bn) {
    case 64: return launch<64, false, false, true>(ta, tb, args, stream);
    case 128: return launch<128, false, false, true>(ta, tb, args, stream);
    default: return launch<256, false, false, true>(ta, tb, args, stream);
  }
}

int gemm_tcgen05_2cta_clamped_glu(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tact, int M, int N, int K, float limit, int* status,
                                  cudaStream_t stream);

// act[M, N] (bfloat16) = clamped GLU of the N gate and N up rows of W against A's rows, where the plain product [M, 2N] would
// take the paired-CTA kernel in whole ranges of K and a tile's 128 gate columns have their up columns; returns 1 elsewhere (the
// narrower tiles that fewer rows take have no such epilogue).
int gemm_bf16_clamped_glu(const void* A, const void* W, __nv_bfloat16* act, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldw, int64_t ld_act,
                          float limit, cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(A) || !a16(W) || !a16(act) || (lda & 7) || (ldw & 7) || (ld_act & 7) || N % 128 != 0 || M < 1 || M > INT32_MAX || 2 * N > INT32_MAX || K < 1 ||
      K > INT32_MAX)
    return 1;
  int bn, splits;
  bool use_pair;
  choose_tile(M, 2 * N, (K + BKH - 1) / BKH, &bn, &splits, &use_pair);
  if (!use_pair || splits != 1) return 1;
  auto map = [](CUtensorMap* m, const void* base, int64_t inner, int64_t outer, int64_t ld, int rows) {
    const uint64_t dims[2] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer)}, strides[1] = {static_cast<uint64_t>(ld) * 2};
    const uint32_t box[2] = {64u, static_cast<uint32_t>(rows)};
    return encode_tensor_map_bf16(m, base, 2, dims, strides, box);
  };
  static_assert(BKH == 64, "boxes of 64 columns");
  CUtensorMap ta, tb, tact;
  int rc = map(&ta, A, K, M, lda, BM);
  if (rc == CTDK_OK) rc = map(&tb, W, K, 2 * N, ldw, 128);
  if (rc == CTDK_OK) rc = map(&tact, act, N, M, ld_act, 32);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  void* const tok = prof_begin(CTDK_PROF_GEMM, 4.0 * static_cast<double>(M) * N * K, stream);
  rc = gemm_tcgen05_2cta_clamped_glu(ta, tb, tact, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), limit, st, stream);
  prof_end(tok, stream);
  return rc;
}

namespace {

template <int OUT>
int launch_out16(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args, cudaStream_t stream) {
  switch (bn) {
    case 64: return launch<64, false, false, true, OUT>(ta, tb, args, stream);
    case 128: return launch<128, false, false, true, OUT>(ta, tb, args, stream);
    default: return launch<256, false, false, true, OUT>(ta, tb, args, stream);
  }
}

}  // namespace

// C (bfloat16) = A B^T with bfloat16 operands, all pitches multiples of 8. up_row > 0: C = silu(gate) up with
// N gate rows of B and their up rows up_row rows further. tiles != null (device memory): the grouped form,
// C[m-block i of 128 rows] = A[m-block i] B[tiles[i]]^T for the first tiles[max_tiles] m-blocks, with group
// g's rows of B from g * n_pitch on; M is then max_tiles * 128.
int gemm_bf16_out16(const void* A, int64_t lda, const void* B, int64_t ldb, __nv_bfloat16* Cp, int64_t ldc, int64_t M, int N, int K, int up_row,
                    const int32_t* tiles, int max_tiles, int64_t n_pitch, int groups, cudaStream_t stream) {
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  CTDK_REQUIRE(a16(A) && a16(B) && a16(Cp) && (lda & 7) == 0 && (ldb & 7) == 0 && (ldc & 7) == 0, "gemm_bf16_out16: operands must be 16-byte aligned");
  const int64_t b_rows = tiles != nullptr ? n_pitch * groups : up_row + N;
  CTDK_REQUIRE(M >= 1 && N >= 1 && K >= 1 && M <= INT32_MAX && b_rows <= INT32_MAX && (tiles == nullptr || n_pitch >= up_row + N),
               "gemm_bf16_out16: bad shape");
  const int cols = up_row > 0 ? 2 * N : N;   // accumulator columns of all tiles
  const int bn = cols >= 256 ? 256 : (cols > 64 ? 128 : 64);
  const uint64_t da[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)}, sa[1] = {static_cast<uint64_t>(lda) * 2};
  const uint64_t db[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(b_rows)}, sb[1] = {static_cast<uint64_t>(ldb) * 2};
  const uint32_t box_a[2] = {static_cast<uint32_t>(BKH), static_cast<uint32_t>(BM)};
  const uint32_t box_b[2] = {static_cast<uint32_t>(BKH), static_cast<uint32_t>(up_row > 0 ? bn / 2 : bn)};
  CUtensorMap ta, tb;
  int rc = encode_tensor_map_bf16(&ta, A, 2, da, sa, box_a);
  if (rc == CTDK_OK) rc = encode_tensor_map_bf16(&tb, B, 2, db, sb, box_b);
  if (rc != CTDK_OK) return rc;
  int* st = device_status_word();
  if (st == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  GemmArgs args{nullptr, nullptr, ldc, static_cast<int>(M), N, K, CTDK_EPI_STORE, 1, 1, st};
  args.tiles = tiles;
  args.max_tiles = max_tiles;
  args.n_pitch = static_cast<int>(n_pitch);
  args.out16 = Cp;
  args.up_row = up_row;
  return up_row > 0 ? launch_out16<kOutGlu>(bn, ta, tb, args, stream) : launch_out16<kOutBf16>(bn, ta, tb, args, stream);
}

// Near-fp32 GEMM (3xTF32 split) is ctdk_gemm_ws; without its workspace the caller takes the exact SIMT kernel.
int gemm_3xtf32(const float*, const float*, float*, int64_t, int64_t, int64_t, int64_t, int64_t,
                int64_t, int, int, int, const float*, cudaStream_t) {
  return 1;
}

// C = A B + A B2 + A2 B (operands split into high and low parts: the 3xTF32 product) in one launch of the cluster kernel.
// The first product is accumulated in runs of at most `run` k-blocks. With more tiles than clusters, or a K whose runs do
// not fit a cluster, the ranges are units of the one-CTA kernel that add their tiles at L2, in an order that shows only
// where it did with three products (K > 1024, or K > 512 with accumulation; in several rounds the
// cluster kernel does not overlap its exchange: 903 rows of SmolLM2-135M 38.4 -> 40.2 ms a step). Returns 1 from about two
// rounds of tiles on: the paired-CTA kernel's large tiles, three times, are then faster.
// The operands are split here, in the launch that as a rule also zeroes C where the product adds to it. Nothing is enqueued when it returns 1.
int gemm_split_tcgen05(const SplitOperands& ops, float* Cp, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int transa,
                       int transb, int epilogue, const float* aux, int run, cudaStream_t stream) {
  const float *A = ops.a_hi, *A2 = ops.a_lo, *B = ops.b_hi, *B2 = ops.b_lo;
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(A) || !a16(B) || !a16(A2) || !a16(B2) || (lda & 3) || (ldb & 3)) return 1;
  if (M < 1 || N < 8 || K < 1 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX / 4) return 1;
  const bool a_mn = transa != 0, b_mn = transb == 0;
  const int64_t k_blocks = (K + BK - 1) / BK;
  const int64_t m_blocks = (M + BM - 1) / BM;
  // the first product's CTAs: as many as its runs need, or its share of the work
  int best_bn = 0, best_s = 0, best_lead = 0;
  double best = 1e300;
  const int widths[2] = {128, 64};
  for (int w : widths)
    for (int S = 2; S <= 8; S *= 2) {
      const int64_t runs = (k_blocks + run - 1) / run;
      const int64_t lead = runs > (S + 2) / 3 ? runs : (S + 2) / 3;
      if (lead >= S || m_blocks * ((N + w - 1) / w) > clusters_of(S) || k_blocks < lead || 2 * k_blocks < S - lead) continue;   // every CTA has a range
      const int64_t longest = std::max((k_blocks + lead - 1) / lead, (2 * k_blocks + S - lead - 1) / (S - lead));
      const double t = static_cast<double>(longest) * (w == 128 ? 0.6 : 0.45) + (w == 128 ? 6.0 : 5.0);
      if (t < best * 0.97) {
        best = t;
        best_bn = w;
        best_s = S;
        best_lead = static_cast<int>(lead);
      }
    }
  int splits = 0, two_runs = 0;
  if (best_s == 0) {
    const int sms = sm_budget();
    const int64_t lead = (k_blocks + run - 1) / run;
    if (m_blocks * ((N + 127) / 128) > 2 * static_cast<int64_t>(sms) || lead > 24) return 1;
    const int wide[2] = {256, 128};
    // Units of two runs where they are one a tile, or two and C is zeroed: the only adds whose order does not show. They
    // give the same bits each time, as the three products one behind the other did.
    two_runs = lead == 1 || (lead == 2 && epilogue != CTDK_EPI_ACCUMULATE) ? 1 : 0;
    for (int w : wide) {
      if (two_runs == 0 || (w == 256 && N <= 128)) continue;
      const double rounds = static_cast<double>((m_blocks * ((N + w - 1) / w) * lead + sms - 1) / sms);
      const int64_t longest = (k_blocks + lead - 1) / lead + (2 * k_blocks + lead - 1) / lead;
      const double t = rounds * (static_cast<double>(longest) + 12.0) * (w == 256 ? 1.0 : 0.6);
      if (t < best * 0.97) {
        best = t;
        best_bn = w;
        splits = static_cast<int>(lead);
      }
    }
    for (int w : wide)
      for (int64_t more = 1; two_runs == 0 && more <= 2 * lead && more <= 2 * k_blocks; ++more) {
        if (w == 256 && N <= 128) break;
        const double rounds = static_cast<double>((m_blocks * ((N + w - 1) / w) * (lead + more) + sms - 1) / sms);
        const int64_t longest = std::max((k_blocks + lead - 1) / lead, (2 * k_blocks + more - 1) / more);
        const double t = rounds * (static_cast<double>(longest) + 12.0) * (w == 256 ? 1.0 : 0.6);
        if (t < best * 0.97) {
          best = t;
          best_bn = w;
          best_lead = static_cast<int>(lead);
          splits = static_cast<int>(lead + more);
        }
      }
  }
  auto map_a = [&](CUtensorMap* m, const float* p) { return a_mn ? make_map(m, p, M, K, lda, BK, true, false) : make_map(m, p, K, M, lda, BM, false, false); };
  auto map_b = [&](CUtensorMap* m, const float* p) {
    return b_mn ? make_map(m, p, N, K, ldb, BK, true, false) : make_map(m, p, K, N, ldb, best_bn, false, false);
  };
  CUtensorMap ta, tb, ta2, tb2;
  int rc = map_a(&ta, A);
  if (rc == CTDK_OK) rc = map_a(&ta2, A2);
  if (rc == CTDK_OK) rc = map_b(&tb, B);
  if (rc == CTDK_OK) rc = map_b(&tb2, B2);
  // The product reads the parts only, so C may be one of the operands: it is then zeroed behind the launch that splits them.
  const float* c_end = Cp + (M - 1) * ldc + N;
  const bool zero = splits > 1 && epilogue != CTDK_EPI_ACCUMULATE;
  const bool in_place = (Cp < ops.a + ops.na && ops.a < c_end) || (Cp < ops.b + ops.nb && ops.b < c_end);
  if (rc == CTDK_OK) rc = split_operands(ops, zero && !in_place ? Cp : nullptr, M, N, ldc, stream);
  if (rc == CTDK_OK && zero && in_place) rc = zero_rows(Cp, M, N, ldc, stream);
  if (rc != CTDK_OK) return rc;
  // the work of the three products, as where they are launched one by one
  void* const tok = prof_begin(CTDK_PROF_GEMM, 6.0 * static_cast<double>(M) * N * K, stream);
  if (splits > 0) {
    GemmArgs g{Cp, aux, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), epilogue, 0, splits, device_status_word()};
    g.vec_ok = a16(Cp) && (ldc & 3) == 0 && (aux == nullptr || a16(aux)) ? 1 : 0;
    g.lead = best_lead;
    g.two_runs = two_runs;
    if (g.status == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
    rc = best_bn == 256 ? dispatch_major<256>(a_mn, b_mn, ta, tb, g, stream, &ta2, &tb2)
                        : dispatch_major<128>(a_mn, b_mn, ta, tb, g, stream, &ta2, &tb2);
    prof_end(tok, stream);
    return rc;
  }
  ClusterArgs c{Cp, aux, ldc, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), epilogue, 0, best_s, 3, best_lead, device_status_word()};
  c.vec_ok = a16(Cp) && (ldc & 3) == 0 && (aux == nullptr || a16(aux)) ? 1 : 0;
  if (c.status == nullptr) return fail(CTDK_ELAUNCH, "gemm: no status word");
  rc = best_bn == 128 ? launch_cluster_major<128>(a_mn, b_mn, ta, tb, ta2, tb2, c, stream)
                      : launch_cluster_major<64>(a_mn, b_mn, ta, tb, ta2, tb2, c, stream);
  prof_end(tok, stream);
  return rc;
}

}  // namespace ctdk
