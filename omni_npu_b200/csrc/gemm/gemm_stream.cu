// Products with few rows, dense, grouped and batched:  C[M,N] = A[M,K] * W[N,K]^T, bf16 in, fp32 accumulate.
//
// What bounds them is the weight stream, so the weights are the M operand: a tile is 128 rows of W times the
// (16 .. 128) rows of A, and a stage of the ring is 16 KB of weights and 2 KB per 16 rows of A.  (With the rows of A
// as the M operand, gemm_tcgen05_kernel, every slab carries 16 KB of A whatever M is.)  A CTA takes half of an SM's
// shared memory: two are resident, or one and the next kernel's, whose first ring of weights then flows while this
// kernel finishes.
//
// Dense: N / 128 tiles; when these are fewer than half the SMs, the 2, 4 or 8 CTAs of a cluster share a tile's
// K and sum their parts in rank order over distributed shared memory.  The split depends on N and K alone, so the
// result of a row does not depend on the number of rows, up to the 128 that the kernel takes; products without a split
// have the same bits on every kernel for bf16 operands (all add up K in steps of 16 in the tensor cores).
// Grouped: tiles of all live experts, each read once; an expert with more rows than a tile takes several tiles side by
// side, which share its weights in L2.
// Batched: the same number of rows for every group, A and C with strides of their own for rows and groups (the heads of
// latent attention, whose queries and results need no transposed copies: 128 rows of 16 heads, 512 x 128, 15.5 us with
// them, 5.8 without).
//
// Measured in a CUDA graph, one row (us, gemm_tcgen05_kernel / here / the weights at 6.4 TB/s): 4096 x 4096
// 17.5 / 9.2 / 5.2, 6144 x 4096 22.7 / 12.5 / 7.8, 4096 x 14336 35.2 / 21.5 / 18.2, 28672 x 4096 with silu 71.5 / 41.4 /
// 36.5, 128256 x 4096 193 / 164 / 163; 83 of 128 experts live, 1536 x 2048 with silu 121 / 83 / 81.
// Against 8 CTAs per cluster throughout: 6144 x 4096 takes 16.0 (only what stays resident at once pays).
//
// Per CTA (192 threads): warp 0 TMA, warp 1 MMA, warps 2-5 epilogue (a thread holds one column of C and the rows of A
// one after another).  Every wait is bounded; on expiry the CTA records a status code, waits for its copies in flight,
// frees its TMEM and returns.

#include "../common/device_once.h"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "column_store.cuh"
#include "group_tiles.cuh"
#include "stream_split.cuh"

namespace b200 {

namespace stream {
constexpr int BW = 128;                  // rows of W per tile
constexpr int SLAB_K = 64;               // elements of K per stage: 128 bytes
constexpr int W_BYTES = BW * 128;
constexpr int THREADS = 192;
constexpr int RING = 108 * 1024;         // of a CTA, so that two fit an SM
constexpr int MAX_EXPERTS = 512;
}  // namespace stream

struct StreamParams {
  int M, N, K;
  int tn;                 // rows of A per tile: 32, 64 or 128; dense 16 too
  int box;                // rows of A per copy: dense tn (rows past the end cost nothing), grouped 16
  int stages, k_slabs, splits, num_n_tiles;
  int num_experts;        // groups (grouped, batched)
  long long c_group;      // batched: elements of C between groups
  int ldc, out_fp32, act;
  int w_ready;            // no kernel still running writes W: its first ring goes ahead of the wait
  float act_alpha, act_limit;
  void* C;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  const int* expert_offsets;
  int* status;
};

struct StreamTile {
  int n0, row0, rows, expert;
};

enum : int { kStreamDense = 0, kStreamGrouped = 1, kStreamBatched = 2 };

template <int MODE>
__device__ __forceinline__ bool stream_tile(const StreamParams& p, const int* prefix, const int* first_row, int t,
                                            int& cursor, StreamTile& tile) {
  if constexpr (MODE == kStreamGrouped) {
    if (t >= prefix[p.num_experts]) return false;
    while (prefix[cursor + 1] <= t) ++cursor;
    const int row0 = first_row[cursor], rows = first_row[cursor + 1] - row0;
    const int row_tiles = (rows + p.tn - 1) / p.tn;
    const int local = t - prefix[cursor], rt = local % row_tiles;
    tile.n0 = local / row_tiles * stream::BW;
    tile.row0 = row0 + rt * p.tn;
    tile.rows = min(p.tn, rows - rt * p.tn);
    tile.expert = cursor;
  } else if constexpr (MODE == kStreamBatched) {
    const int row_tiles = (p.M + p.tn - 1) / p.tn, per_group = row_tiles * p.num_n_tiles;
    tile.expert = t / per_group;
    if (tile.expert >= p.num_experts) return false;
    const int local = t - tile.expert * per_group, rt = local % row_tiles;
    tile.n0 = local / row_tiles * stream::BW;
    tile.row0 = rt * p.tn;
    tile.rows = min(p.tn, p.M - tile.row0);
  } else {
    if (t >= p.num_n_tiles) return false;
    tile.n0 = t * stream::BW;
    tile.row0 = 0;
    tile.rows = p.M;
    tile.expert = 0;
  }
  return true;
}

// One value of C per thread (column n; the 32 lanes of a warp hold neighbouring columns): epilogue and store.
__device__ __forceinline__ void stream_store(const StreamParams& p, int act, float v, int row, int n) {
  const bool ok = n < p.N;
  const float bias = p.bias && ok ? __bfloat162float(p.bias[n]) : 0.f;
  if (act_is_gated(act)) {
    v += bias;
    // columns alternate in groups of eight: gate, up (N is a multiple of 16)
    const float up = __shfl_xor_sync(0xffffffffu, v, 8);
    if (ok && !(n & 8))
      static_cast<__nv_bfloat16*>(p.C)[static_cast<size_t>(row) * p.ldc + (n >> 4) * 8 + (n & 7)] =
          __float2bfloat16(gated_act(act, v, up, p.act_alpha, p.act_limit));
    return;
  }
  if (act_is_unary(act)) v = unary_act(act, v, p.act_alpha, p.act_limit);
  if (!ok) return;
  v += bias;
  const size_t at = static_cast<size_t>(row) * p.ldc + n;
  if (p.residual) v += __bfloat162float(p.residual[at]);
  if (p.out_fp32)
    static_cast<float*>(p.C)[at] = v;
  else
    static_cast<__nv_bfloat16*>(p.C)[at] = __float2bfloat16(v);
}

// Four neighbouring values of a row per lane (column n, a multiple of four).  wide: C, the residual and their pitch let
// four values be one access.
__device__ __forceinline__ void stream_store4(const StreamParams& p, int act, float (&v)[4], int row, int n, bool wide) {
  const bool gated = act_is_gated(act), whole = n + 3 < p.N;
  if (act_is_unary(act))
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = unary_act(act, v[i], p.act_alpha, p.act_limit);
  if (p.bias)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < p.N) v[i] += __bfloat162float(p.bias[n + i]);
  size_t at = static_cast<size_t>(row) * p.ldc + n;
  if (gated) {
    // columns alternate in groups of eight: gate, up (N is a multiple of 16); the lane after the next has the up columns
    float up[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) up[i] = __shfl_xor_sync(0xffffffffu, v[i], 2);
    if (!whole || (n & 8)) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = gated_act(act, v[i], up[i], p.act_alpha, p.act_limit);
    at = static_cast<size_t>(row) * p.ldc + (n >> 4) * 8 + (n & 7);
  }
  if (wide && whole) {
    if (p.residual) {
      const uint2 r = *reinterpret_cast<const uint2*>(p.residual + at);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
      v[0] += a.x, v[1] += a.y, v[2] += b.x, v[3] += b.y;
    }
    if (p.out_fp32)
      *reinterpret_cast<float4*>(static_cast<float*>(p.C) + at) = make_float4(v[0], v[1], v[2], v[3]);
    else
      *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.C) + at) =
          make_uint2(columns_pack(v[0], v[1]), columns_pack(v[2], v[3]));
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (n + i >= p.N) break;
    if (p.residual) v[i] += __bfloat162float(p.residual[at + i]);
    if (p.out_fp32)
      static_cast<float*>(p.C)[at + i] = v[i];
    else
      static_cast<__nv_bfloat16*>(p.C)[at + i] = __float2bfloat16(v[i]);
  }
}

// SPLIT: the CTAs of a cluster share a tile's K.  ACT: p.act is looked at.  (With every activation's code the
// unsplit kernels take 168 registers, which leave the kernel behind no room beside two of their CTAs, without it 113 to 137:
// latent decode step of 128 rows, 4 layers, 1334 us with one kernel for all, 1312.)
template <int MODE, bool SPLIT, bool ACT>
__global__ void __launch_bounds__(stream::THREADS, 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                   const StreamParams p) {
  using namespace stream;
  constexpr bool GROUPED = MODE == kStreamGrouped, BATCHED = MODE == kStreamBatched;
  const int act = ACT ? p.act : static_cast<int>(kActNone);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int stage_bytes = W_BYTES + p.tn * 128;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty_bar = full_bar + p.stages;
  uint64_t* tmem_full = empty_bar + p.stages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* drain_bar = tmem_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* prefix = const_cast<int*>(abort_flag) + 1;       // grouped: tiles before an expert, [E + 1]
  int* first_row = prefix + p.num_experts + 1;          // grouped: the offsets

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int acc_stride = p.tn;
  const uint32_t tmem_cols = p.tn < 32 ? 32u : 2u * p.tn;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 4);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  if constexpr (GROUPED) {
    pdl_wait();      // the offsets come from an earlier kernel
    if (warp == 2)
      group_tiles(p.expert_offsets, p.num_experts, prefix, first_row,
                  [&](int rows) { return (rows + p.tn - 1) / p.tn * p.num_n_tiles; });
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int t_first = SPLIT ? blockIdx.x / p.splits : blockIdx.x, t_stride = SPLIT ? gridDim.x / p.splits : gridDim.x;
  const int per = SPLIT ? (p.k_slabs + p.splits - 1) / p.splits : p.k_slabs;
  const int k_begin = rank * per, k_end = min(p.k_slabs, k_begin + per);

  pdl_trigger();
  // weights that no kernel ahead of this one writes (the caller says so): their first ring is under way before the wait
  const bool early = !GROUPED && p.w_ready && threadIdx.x == 0;
  if (!early) pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0, cursor = 0, preloaded = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      StreamTile tile;
      if (early) {
        if (stream_tile<MODE>(p, prefix, first_row, t_first, cursor, tile)) {
          const uint32_t bytes = W_BYTES + (tile.rows + p.box - 1) / p.box * p.box * 128;
          for (; preloaded < p.stages && k_begin + preloaded < k_end; ++preloaded) {
            mbar_arrive_expect_tx(&full_bar[preloaded], bytes);
            if constexpr (BATCHED)
              tma_load_3d(smem + preloaded * stage_bytes, &tm_w, &full_bar[preloaded], (k_begin + preloaded) * SLAB_K,
                          tile.n0, tile.expert);
            else
              tma_load_2d(smem + preloaded * stage_bytes, &tm_w, &full_bar[preloaded], (k_begin + preloaded) * SLAB_K,
                          tile.n0);
          }
        }
        pdl_wait();
      }
      for (int t = t_first; ok && stream_tile<MODE>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        const int boxes = (tile.rows + p.box - 1) / p.box;
        for (int k = k_begin; k < k_end; ++k) {
          uint8_t* dst = smem + stage * stage_bytes;
          if (issued >= preloaded) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
              atomicCAS(p.status, 0, kStatusTimeoutEmptyBarrier);
              *abort_flag = 1;
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>(W_BYTES + boxes * p.box * 128));
            if constexpr (GROUPED || BATCHED)
              tma_load_3d(dst, &tm_w, &full_bar[stage], k * SLAB_K, tile.n0, tile.expert);
            else
              tma_load_2d(dst, &tm_w, &full_bar[stage], k * SLAB_K, tile.n0);
          }
          for (int i = 0; i < boxes; ++i) {
            if constexpr (BATCHED)
              tma_load_3d(dst + W_BYTES + i * p.box * 128, &tm_x, &full_bar[stage], k * SLAB_K, tile.row0 + i * p.box,
                          tile.expert);
            else
              tma_load_2d(dst + W_BYTES + i * p.box * 128, &tm_x, &full_bar[stage], k * SLAB_K, tile.row0 + i * p.box);
          }
          ++issued;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        // (only after the first ring, so every stage's last copies are complete sets): wait, bounded, until they land
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < p.stages && i < issued; ++i) {
          if (--s < 0) {
            s = p.stages - 1;
            ph ^= 1;
          }
          mbar_wait(&full_bar[s], ph);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0, cursor = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      StreamTile tile;
      const uint32_t lo0 = (smem_u32(smem) & 0x3FFFF) >> 4;
      for (int t = t_first; ok && stream_tile<MODE>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        if (*abort_flag || !mbar_wait(&tmem_empty[acc], acc_phase ^ 1)) {
          if (!*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemEmpty);
          *abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t idesc = make_idesc(1, 1, BW, (tile.rows + p.box - 1) / p.box * p.box);
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * acc_stride);
        for (int k = k_begin; k < k_end; ++k) {
          if (!mbar_wait(&full_bar[stage], phase)) {
            atomicCAS(p.status, 0, kStatusTimeoutFullBarrier);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t w_lo = lo0 + ((stage * stage_bytes) >> 4), x_lo = w_lo + (W_BYTES >> 4);
          umma_first<kKindBF16>(d, w_lo, x_lo, idesc, k > k_begin ? 1u : 0u);
          umma_acc<kKindBF16>(d, w_lo + 2, x_lo + 2, idesc);
          umma_acc<kKindBF16>(d, w_lo + 4, x_lo + 4, idesc);
          umma_acc<kKindBF16>(d, w_lo + 6, x_lo + 6, idesc);
          tc_commit(&empty_bar[stage]);
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit(&tmem_full[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;      // row of the W tile
    // bf16 results without a residual, and without a bias behind a unary activation: stored in pairs of columns
    const bool plain = !p.out_fp32 && !p.residual && !(p.bias && act_is_unary(act));
    const bool pairs = columns_pair(p.C, p.ldc | (BATCHED ? p.c_group : 0), p.N, act_is_gated(act));
    const bool plain32 = MODE == kStreamDense && p.out_fp32 && !p.residual && act == kActNone;
    int cursor = 0, acc = 0;
    uint32_t acc_phase = 0;
    StreamTile tile;
    for (int t = t_first; stream_tile<MODE>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
      bool ok = !*abort_flag && mbar_wait(&tmem_full[acc], acc_phase);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0 && !*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemFull);
        *abort_flag = 1;
        break;
      }
      tc_fence_after_sync();
      const uint32_t col = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * acc_stride);
      const int col_n = tile.n0 + r;
      const float bias = (plain || plain32) && p.bias && col_n < p.N ? __bfloat162float(p.bias[col_n]) : 0.f;
      float* part = reinterpret_cast<float*>(smem);      // split K: [row of A][128] (the ring has been read)
      for (int c = 0; c < tile.rows; c += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(col + static_cast<uint32_t>(c))
            : "memory");
        tmem_ld_wait();
        const int n = min(16, tile.rows - c);
        if constexpr (SPLIT) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < n) part[(c + i) * BW + r] = __uint_as_float(v[i]);
        } else if (plain) {
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]) + bias;
          store_act_columns(act, p.act_alpha, p.act_limit, x,
                            static_cast<__nv_bfloat16*>(p.C) + (BATCHED ? tile.expert * p.c_group : 0) +
                                static_cast<size_t>(tile.row0 + c) * p.ldc,
                            p.ldc, col_n, p.N, n, pairs);
        } else if (plain32) {
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]) + bias;
          store_fp32_columns(x, static_cast<float*>(p.C) + static_cast<size_t>(tile.row0 + c) * p.ldc, p.ldc, col_n, p.N, n);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < n) stream_store(p, act, __uint_as_float(v[i]), tile.row0 + c + i, col_n);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if constexpr (SPLIT) {
    // one tile per CTA: the CTAs of the cluster share out its rows of A, a row per warp and four columns per lane (a row
    // takes some 0.28 us, the latency of the other CTAs' shared memory: 63 rows of 2048 x 512 in two parts took 13.9 us
    // with all warps on one row, 7.4 in this form)
    cluster_sync_all();
    if (warp >= 2 && !*abort_flag) {
      const int n = t_first * BW + 4 * lane;
      const bool wide = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & (p.out_fp32 ? 15 : 7)) == 0 &&
                        (reinterpret_cast<uintptr_t>(p.residual) & 7) == 0;
      for (int row = rank + p.splits * (warp - 2); row < p.M; row += 4 * p.splits) {
        const uint32_t at = smem_u32(smem) + static_cast<uint32_t>((row * BW + 4 * lane) * 4);
        float sum[4];
        split_sum(at, p.splits, sum);
        stream_store4(p, act, sum, row, n, wide);
      }
    }
    cluster_sync_all();
  }
  if (warp == 1) {
    if (*abort_flag && lane == 0) {
      // products still in flight write tensor memory: wait (bounded) for them before it is freed
      tc_commit(drain_bar);
      mbar_wait(drain_bar, 0);
    }
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

static int stream_stages(int tn) {
  const int n = stream::RING / (stream::W_BYTES + tn * 128);
  return n > 8 ? 8 : n;
}

static size_t stream_smem(int tn, int stages, int num_experts) {
  return 1024 + static_cast<size_t>(stages) * (stream::W_BYTES + tn * 128) + (2 * stages + 5) * 8 + 8 +
         (num_experts > 0 ? 2 * (num_experts + 1) * 4 : 0);
}

template <int MODE, bool SPLIT, bool ACT>
static int launch_stream(const CUtensorMap& tw, const CUtensorMap& tx, const StreamParams& p, int grid,
                         cudaStream_t stream) {
  auto kern = gemm_stream_kernel<MODE, SPLIT, ACT>;
  static DeviceOnce once;
  int dev = 0;
  if (once.needed(&dev)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024) != cudaSuccess) return -20;
    once.mark(dev);
  }
  return launch_pdl(kern, dim3(grid), dim3(stream::THREADS), stream_smem(p.tn, p.stages, MODE == kStreamGrouped ? p.num_experts : 0), stream,
                    p.splits, tw, tx, p) == cudaSuccess
             ? 0
             : -21;
}

}  // namespace b200

using namespace b200;

// CTAs of a cluster that b200_gemm_stream has share the K of one tile.  None where one CTA on half the SMs takes in what
// the memory gives, nor for short rows, where the exchange costs what the split gains (us, no split / two parts, with 1 and
// 64 rows: 12288 x 2048 with silu 13.4 / 13.9 and 15.9 / 19.9, 16384 x 2048 14.4 / 14.6 and 16.9 / 18.2, 18944 x 4096
// 30.8 / 27.7 and 34.2 / 31.7, 2048 x 512 5.0 / 4.7 and 7.0 / 7.5).
extern "C" int b200_gemm_stream_splits(int N, int K, int max_ctas, int sms) {
  const int tiles = (N + stream::BW - 1) / stream::BW, slabs = (K + stream::SLAB_K - 1) / stream::SLAB_K;
  return 2 * tiles > sms || slabs <= 8 ? 1 : stream_splits(tiles, slabs, max_ctas, sms);
}

// A [M <= 128, K] (pitch lda), W [N, K] (pitch ldw), C [M, N, or N / 2 with a gated activation].
// w_ready: see StreamParams.
extern "C" int b200_gemm_stream(const void* A, const void* W, void* C, const void* bias, const void* residual, int M,
                                int N, int K, int lda, int ldw, int ldc, int out_fp32, int act, int* status,
                                int max_ctas, float act_alpha, float act_limit, int w_ready, cudaStream_t cu_stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 128) return -10;
  if (act_is_gated(act) && ((N % 16) != 0 || out_fp32 || residual)) return -11;
  StreamParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.tn = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  p.box = p.tn;
  p.stages = stream_stages(p.tn);
  p.k_slabs = (K + stream::SLAB_K - 1) / stream::SLAB_K;
  p.num_n_tiles = (N + stream::BW - 1) / stream::BW;
  p.splits = b200_gemm_stream_splits(N, K, max_ctas, sm_count());
  p.ldc = ldc;
  p.out_fp32 = out_fp32;
  p.act = act;
  p.w_ready = w_ready;
  p.act_alpha = act_alpha;
  p.act_limit = act_limit;
  p.C = C;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.status = status;
  CUtensorMap tw, tx;
  int r = make_tensormap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, N, K, ldw, stream::BW, stream::SLAB_K,
                            CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  r = make_tensormap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, M, K, lda, p.box, stream::SLAB_K,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  int grid = p.num_n_tiles * p.splits;
  if (p.splits == 1) {
    const int most = max_ctas > 0 ? max_ctas : 2 * sm_count();
    if (grid > most) grid = most;
  }
  if (act == kActNone)
    return p.splits > 1 ? launch_stream<kStreamDense, true, false>(tw, tx, p, grid, cu_stream)
                        : launch_stream<kStreamDense, false, false>(tw, tx, p, grid, cu_stream);
  return p.splits > 1 ? launch_stream<kStreamDense, true, true>(tw, tx, p, grid, cu_stream)
                      : launch_stream<kStreamDense, false, true>(tw, tx, p, grid, cu_stream);
}

// A [total_rows, K], W [E, N, K]; rows expert_offsets[e] .. expert_offsets[e + 1] (device) belong to expert e.
// tn: rows of A per tile, 32, 64 or 128.
extern "C" int b200_grouped_gemm_stream(const void* A, const void* W, void* C, const int* expert_offsets,
                                        int num_experts, int total_rows, int N, int K, int lda, int ldc, int act, int tn,
                                        int* status, int max_ctas, float act_alpha, float act_limit,
                                        cudaStream_t cu_stream) {
  if (total_rows <= 0 || num_experts <= 0 || N <= 0 || K <= 0) return 0;
  if (num_experts > stream::MAX_EXPERTS) return -13;
  if (tn != 32 && tn != 64 && tn != 128) return -10;
  if (act_is_gated(act) && (N % 16) != 0) return -11;
  StreamParams p{};
  p.M = total_rows;
  p.N = N;
  p.K = K;
  p.tn = tn;
  p.box = 16;
  p.stages = stream_stages(tn);
  p.k_slabs = (K + stream::SLAB_K - 1) / stream::SLAB_K;
  p.num_n_tiles = (N + stream::BW - 1) / stream::BW;
  p.splits = 1;
  p.num_experts = num_experts;
  p.ldc = ldc;
  p.act = act;
  p.act_alpha = act_alpha;
  p.act_limit = act_limit;
  p.C = C;
  p.expert_offsets = expert_offsets;
  p.status = status;
  // at most one row tile per expert beyond those that total_rows fill
  const long long row_tiles = total_rows / tn + (num_experts < total_rows ? num_experts : total_rows);
  if (row_tiles * p.num_n_tiles > 0x7fffffffll) return -14;
  CUtensorMap tw, tx;
  int r = make_tensormap_3d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, num_experts, N, K, static_cast<uint64_t>(N) * K,
                            K, stream::BW, stream::SLAB_K, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  r = make_tensormap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, total_rows, K, lda, p.box, stream::SLAB_K,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  int grid = max_ctas > 0 ? max_ctas : 2 * sm_count();
  if (row_tiles * p.num_n_tiles < grid) grid = static_cast<int>(row_tiles * p.num_n_tiles);
  return act == kActNone ? launch_stream<kStreamGrouped, false, false>(tw, tx, p, grid, cu_stream)
                         : launch_stream<kStreamGrouped, false, true>(tw, tx, p, grid, cu_stream);
}

// C[t, g, :] = A[t, g, :] W[g]^T for T rows of G groups: A and C with pitches of their own between rows and groups (in
// elements), W [G, N, K].  Returns 1 (nothing done) for pitches and alignments that the copies do not take.
extern "C" int b200_batched_gemm(const void* A, const void* W, void* C, int T, int G, int N, int K, long long a_row,
                                 long long a_group, long long c_row, long long c_group, int tn, int* status, int w_ready,
                                 cudaStream_t cu_stream) {
  if (T <= 0 || G <= 0 || N <= 0 || K <= 0) return 0;
  if (tn != 32 && tn != 64 && tn != 128) return -10;
  if (((a_row | a_group | K) & 7) != 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) != 0 ||
      a_row <= 0 || (G > 1 && a_group <= 0) || c_row > 0x7fffffffll)
    return 1;
  StreamParams p{};
  p.M = T;
  p.N = N;
  p.K = K;
  p.tn = tn;
  p.box = tn;
  p.stages = stream_stages(tn);
  p.k_slabs = (K + stream::SLAB_K - 1) / stream::SLAB_K;
  p.num_n_tiles = (N + stream::BW - 1) / stream::BW;
  p.splits = 1;
  p.num_experts = G;
  p.c_group = c_group;
  p.w_ready = w_ready;
  p.ldc = static_cast<int>(c_row);
  p.C = C;
  p.status = status;
  const long long tiles = static_cast<long long>(G) * p.num_n_tiles * ((T + tn - 1) / tn);
  if (tiles > 0x3fffffffll) return -14;
  CUtensorMap tw, tx;
  int r = make_tensormap_3d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, G, N, K, static_cast<uint64_t>(N) * K, K,
                            stream::BW, stream::SLAB_K, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  r = make_tensormap_3d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, G, T, K, static_cast<uint64_t>(G > 1 ? a_group : K),
                        static_cast<uint64_t>(a_row), p.box, stream::SLAB_K, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  const int grid = tiles < 2 * sm_count() ? static_cast<int>(tiles) : 2 * sm_count();
  return launch_stream<kStreamBatched, false, false>(tw, tx, p, grid, cu_stream);
}
