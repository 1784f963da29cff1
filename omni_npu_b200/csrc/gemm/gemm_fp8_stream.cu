// Block-scaled e4m3 products with few rows, dense and grouped (the operands and scales of gemm_fp8_block.cu):
//
//   C[m, n] = sum_kb  a_s[m, kb] * w_s[n / 128, kb] * sum_{k in block kb} A[m, k] * W[n, k]
//
// What bounds them is the weight stream, so the weights are the M operand, as in gemm_stream.cu: a tile is 128 rows of W
// times 16 to 64 rows of A, a stage of the ring one scale block of K (16 KB of weights and 2 KB per 16 rows of A), and
// two CTAs share an SM.  Every stage's product goes to a fresh accumulator of four in tensor memory; a thread of the
// epilogue holds one row of W and adds the accumulator's columns, scaled, to its fp32 sums.  The rows' scales are
// loaded one per lane, a stage ahead, and passed around by shuffles.
//
// Dense: when the tiles are fewer than the resident CTAs, the 2, 4 or 8 CTAs of a cluster share a tile's K and sum their
// parts in rank order; the split depends on N and K alone, so that up to 64 rows the result of a row does not depend on the
// others (gemm_fp8_block.cu, beyond, has no split).  Grouped: tiles of all live experts.
//
// Measured in a CUDA graph (us, gemm_fp8_block_kernel / here / the weights at 6.4 TB/s): one row 4096 x 7168
// 31.8 / 10.2 / 4.6, 18432 x 7168 41.4 / 25.1 / 20.5; 32 experts, 32 rows each, 4096 x 7168 with silu 214 / 159 / 146,
// 7168 x 2048 111 / 88 / 73.  Tiles of 32 rows take as long as those of 64 up to 16 rows per expert, and longer beyond.
//
// Per CTA (192 threads): warp 0 TMA, warp 1 MMA, warps 2-5 epilogue.  Every wait is bounded; on expiry the CTA records a
// status code, waits for its copies in flight, frees its TMEM and returns.

#include "../common/device_once.h"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "column_store.cuh"
#include "group_tiles.cuh"
#include "stream_split.cuh"

namespace b200 {

namespace fp8s {
constexpr int BW = 128;                  // rows of W per tile
constexpr int SLAB = 128;                // elements (bytes) of K per stage: one scale block
constexpr int W_BYTES = BW * SLAB;
constexpr int MAX_ROWS = 64;             // rows of A per tile
constexpr int PARTS = 4;                 // accumulators in tensor memory
constexpr int THREADS = 192;
constexpr int RING = 108 * 1024;
constexpr int MAX_EXPERTS = 512;
}  // namespace fp8s

struct Fp8StreamParams {
  int M, N, k_slabs;
  int tn, box, stages, splits, num_n_tiles, num_experts, scale_rows, up_scale_row0, ldc, out_fp32, swiglu;
  int w_ready;                // dense: no kernel still running writes W, its first ring goes ahead of the wait
  const float* a_scales;      // [rows, k_slabs]
  const float* w_scales;      // [E][scale_rows, k_slabs]
  void* C;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  const int* expert_offsets;
  int* status;
};

struct Fp8StreamTile {
  int n0, row0, rows, expert;
};

template <bool GROUPED>
__device__ __forceinline__ bool fp8_stream_tile(const Fp8StreamParams& p, const int* prefix, const int* first_row, int t,
                                                int& cursor, Fp8StreamTile& tile) {
  if constexpr (GROUPED) {
    if (t >= prefix[p.num_experts]) return false;
    while (prefix[cursor + 1] <= t) ++cursor;
    const int row0 = first_row[cursor], rows = first_row[cursor + 1] - row0;
    const int row_tiles = (rows + p.tn - 1) / p.tn;
    const int local = t - prefix[cursor], rt = local % row_tiles;
    tile.n0 = local / row_tiles * fp8s::BW;
    tile.row0 = row0 + rt * p.tn;
    tile.rows = min(p.tn, rows - rt * p.tn);
    tile.expert = cursor;
  } else {
    if (t >= p.num_n_tiles) return false;
    tile.n0 = t * fp8s::BW;
    tile.row0 = 0;
    tile.rows = p.M;
    tile.expert = 0;
  }
  return true;
}

// TN: rows of A that the registers have room for (p.tn <= TN).  SPLIT: the CTAs of a cluster share a tile's K.
template <int TN, bool GROUPED, bool SPLIT>
__global__ void __launch_bounds__(fp8s::THREADS, 2)
gemm_fp8_stream_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                       const Fp8StreamParams p) {
  using namespace fp8s;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int stage_bytes = W_BYTES + TN * SLAB;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty_bar = full_bar + p.stages;
  uint64_t* part_full = empty_bar + p.stages;           // [PARTS]
  uint64_t* part_empty = part_full + PARTS;
  uint64_t* drain_bar = part_empty + PARTS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* prefix = const_cast<int*>(abort_flag) + 1;       // grouped: tiles before an expert, [E + 1]
  int* first_row = prefix + p.num_experts + 1;          // grouped: the offsets
  constexpr uint32_t kTmemCols = PARTS * TN;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < PARTS; ++i) {
      mbar_init(&part_full[i], 1);
      mbar_init(&part_empty[i], 4);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
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
      Fp8StreamTile tile;
      if (early) {
        if (fp8_stream_tile<GROUPED>(p, prefix, first_row, t_first, cursor, tile)) {
          const uint32_t bytes = W_BYTES + (tile.rows + p.box - 1) / p.box * p.box * SLAB;
          for (; preloaded < p.stages && k_begin + preloaded < k_end; ++preloaded) {
            mbar_arrive_expect_tx(&full_bar[preloaded], bytes);
            tma_load_2d(smem + preloaded * stage_bytes, &tm_w, &full_bar[preloaded], (k_begin + preloaded) * SLAB, tile.n0);
          }
        }
        pdl_wait();
      }
      for (int t = t_first; ok && fp8_stream_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
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
            mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>(W_BYTES + boxes * p.box * SLAB));
            if constexpr (GROUPED)
              tma_load_3d(dst, &tm_w, &full_bar[stage], k * SLAB, tile.n0, tile.expert);
            else
              tma_load_2d(dst, &tm_w, &full_bar[stage], k * SLAB, tile.n0);
          }
          for (int i = 0; i < boxes; ++i)
            tma_load_2d(dst + W_BYTES + i * p.box * SLAB, &tm_x, &full_bar[stage], k * SLAB, tile.row0 + i * p.box);
          ++issued;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        // (only after the first ring, so every stage's last copies are complete sets): wait, bounded, until they land
        for (int i = 0; i < p.stages && i < issued; ++i) {
          if (--stage < 0) {
            stage = p.stages - 1;
            phase ^= 1;
          }
          mbar_wait(&full_bar[stage], phase);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0, cursor = 0, part = 0;
      uint32_t phase = 0, part_phase = 0;
      bool ok = true;
      Fp8StreamTile tile;
      const uint32_t lo0 = (smem_u32(smem) & 0x3FFFF) >> 4;
      for (int t = t_first; ok && fp8_stream_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        const uint32_t idesc = make_idesc(0, 0, BW, (tile.rows + 15) & ~15);          // e4m3 x e4m3 -> fp32
        for (int k = k_begin; k < k_end; ++k) {
          if (!mbar_wait(&part_empty[part], part_phase ^ 1) || !mbar_wait(&full_bar[stage], phase)) {
            if (!*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutFullBarrier);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t d = tmem_base + static_cast<uint32_t>(part * TN);
          const uint32_t w_lo = lo0 + ((stage * stage_bytes) >> 4), x_lo = w_lo + (W_BYTES >> 4);
          umma_first<kKindFP8>(d, w_lo, x_lo, idesc, 0u);
          umma_acc<kKindFP8>(d, w_lo + 2, x_lo + 2, idesc);
          umma_acc<kKindFP8>(d, w_lo + 4, x_lo + 4, idesc);
          umma_acc<kKindFP8>(d, w_lo + 6, x_lo + 6, idesc);
          tc_commit(&empty_bar[stage]);
          tc_commit(&part_full[part]);
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
          if (++part == PARTS) {
            part = 0;
            part_phase ^= 1;
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ scaling, sums, epilogue
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;      // row of the W tile
    const bool plain = !p.out_fp32 && !p.residual;
    const bool pairs = columns_pair(p.C, p.ldc, p.N, p.swiglu != 0);
    int cursor = 0, part = 0;
    uint32_t part_phase = 0;
    bool ok = true;
    Fp8StreamTile tile;
    for (int t = t_first; ok && fp8_stream_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
      const int n = tile.n0 + r;
      // scale row of this row of W; gate and up rows alternate in groups of eight, their scale rows do not
      const int sn = min(n, p.N - 1);
      const int s_row = !p.swiglu ? sn / 128 : ((sn & 8) ? p.up_scale_row0 : 0) + (sn >> 1) / 128;
      const float* w_s = p.w_scales + (static_cast<long long>(tile.expert) * p.scale_rows + s_row) * p.k_slabs;
      const float* a_s = p.a_scales + static_cast<long long>(tile.row0) * p.k_slabs;
      const bool lo_ok = lane < tile.rows, hi_ok = TN > 32 && lane + 32 < tile.rows;
      const float* a_lo = a_s + static_cast<long long>(lo_ok ? lane : 0) * p.k_slabs;
      const float* a_hi = a_s + static_cast<long long>(hi_ok ? lane + 32 : 0) * p.k_slabs;
      float acc[TN];
#pragma unroll
      for (int c = 0; c < TN; ++c) acc[c] = 0.f;
      float w_n = w_s[k_begin], lo_n = a_lo[k_begin], hi_n = TN > 32 ? a_hi[k_begin] : 0.f;
      for (int k = k_begin; k < k_end; ++k) {
        const float w = w_n, lo = lo_n, hi = hi_n;
        if (k + 1 < k_end) {           // the next stage's scales are on their way while this one is added
          w_n = w_s[k + 1];
          lo_n = a_lo[k + 1];
          if (TN > 32) hi_n = a_hi[k + 1];
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&part_full[part], part_phase))) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t col = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(part * TN);
#pragma unroll
        for (int h = 0; h < TN / 32; ++h) {
          if (h * 32 >= tile.rows) break;
          uint32_t v[32];
          tmem_ld_32x32b_x32(col + h * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const float s = __shfl_sync(0xffffffffu, h ? hi : lo, c) * w;
            acc[h * 32 + c] = fmaf(s, __uint_as_float(v[c]), acc[h * 32 + c]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&part_empty[part]);
        if (++part == PARTS) {
          part = 0;
          part_phase ^= 1;
        }
      }
      if (!ok) break;
      if constexpr (SPLIT) {
        float* sums = reinterpret_cast<float*>(smem);      // [row of A][128]; the ring has been read
#pragma unroll
        for (int c = 0; c < TN; ++c)
          if (c < tile.rows) sums[c * BW + r] = acc[c];
      } else {
        const float bias = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
#pragma unroll
        for (int c = 0; c < TN; c += 16) {
          if (c >= tile.rows) break;
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = acc[c + i] + bias;
          const size_t at = static_cast<size_t>(tile.row0 + c) * p.ldc;
          if (plain) {
            store_act_columns(p.swiglu ? kActSilu : kActNone, 0.f, 0.f, x, static_cast<__nv_bfloat16*>(p.C) + at, p.ldc, n,
                              p.N, tile.rows - c, pairs);
          } else if (n < p.N) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (c + i >= tile.rows) break;
              const size_t o = at + static_cast<size_t>(i) * p.ldc + n;
              const float y = x[i] + (p.residual ? __bfloat162float(p.residual[o]) : 0.f);
              if (p.out_fp32)
                static_cast<float*>(p.C)[o] = y;
              else
                static_cast<__nv_bfloat16*>(p.C)[o] = __float2bfloat16(y);
            }
          }
        }
      }
    }
    if (!ok && lane == 0) {
      if (!*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemFull);
      *abort_flag = 1;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if constexpr (SPLIT) {
    // one tile per CTA: the CTAs of the cluster share out its rows of A, a row per warp and four columns per lane
    // (gemm_stream.cu; 64 rows of 4096 x 1024 in two parts 12.4 us with all warps on one row, 8.2)
    cluster_sync_all();
    if (warp >= 2 && !*abort_flag) {
      const int n = t_first * BW + 4 * lane;
      float bias[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) bias[i] = p.bias && n + i < p.N ? __bfloat162float(p.bias[n + i]) : 0.f;
      const bool wide = n + 3 < p.N && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & (p.out_fp32 ? 15 : 7)) == 0;
      for (int row = rank + p.splits * (warp - 2); row < p.M; row += 4 * p.splits) {
        const uint32_t at = smem_u32(smem) + static_cast<uint32_t>((row * BW + 4 * lane) * 4);
        const size_t o = static_cast<size_t>(row) * p.ldc + n;
        float sum[4];
        split_sum(at, p.splits, sum);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sum[i] += bias[i];
          if (p.residual && n + i < p.N) sum[i] += __bfloat162float(p.residual[o + i]);
        }
        if (wide && p.out_fp32) {
          *reinterpret_cast<float4*>(static_cast<float*>(p.C) + o) = make_float4(sum[0], sum[1], sum[2], sum[3]);
        } else if (wide) {
          *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.C) + o) =
              make_uint2(columns_pack(sum[0], sum[1]), columns_pack(sum[2], sum[3]));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (n + i >= p.N) break;
            if (p.out_fp32)
              static_cast<float*>(p.C)[o + i] = sum[i];
            else
              static_cast<__nv_bfloat16*>(p.C)[o + i] = __float2bfloat16(sum[i]);
          }
        }
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
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int TN, bool GROUPED, bool SPLIT>
static int launch_fp8_stream(const CUtensorMap& tw, const CUtensorMap& tx, const Fp8StreamParams& p, int grid,
                             cudaStream_t stream) {
  auto kern = gemm_fp8_stream_kernel<TN, GROUPED, SPLIT>;
  static DeviceOnce once;
  int dev = 0;
  if (once.needed(&dev)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024) != cudaSuccess) return -20;
    once.mark(dev);
  }
  const size_t smem = 1024 + static_cast<size_t>(p.stages) * (fp8s::W_BYTES + TN * fp8s::SLAB) +
                      (2 * p.stages + 2 * fp8s::PARTS + 1) * 8 + 8 + (GROUPED ? 2 * (p.num_experts + 1) * 4 : 0);
  return launch_pdl(kern, dim3(grid), dim3(fp8s::THREADS), smem, stream, SPLIT ? p.splits : 1, tw, tx, p) == cudaSuccess
             ? 0
             : -21;
}

}  // namespace b200

using namespace b200;

// The operands of b200_gemm_fp8_block, at most 64 rows.  w_ready: see Fp8StreamParams.
extern "C" int b200_gemm_fp8_stream(const void* A, const float* a_scales, const void* W, const float* w_scales, void* C,
                                    const void* bias, const void* residual, int M, int N, int K, int lda, int ldw, int ldc,
                                    int out_fp32, int* status, int max_ctas, int w_ready, cudaStream_t stream) {
  using namespace fp8s;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > MAX_ROWS || (K % SLAB) != 0) return -10;
  Fp8StreamParams p{};
  p.M = M;
  p.N = N;
  p.k_slabs = K / SLAB;
  p.tn = M <= 32 ? 32 : 64;
  p.box = p.tn;
  p.stages = RING / (W_BYTES + p.tn * SLAB);
  p.num_n_tiles = (N + BW - 1) / BW;
  p.splits = stream_splits(p.num_n_tiles, p.k_slabs, max_ctas, sm_count());
  p.scale_rows = p.num_n_tiles;
  p.ldc = ldc;
  p.out_fp32 = out_fp32;
  p.w_ready = w_ready;
  p.a_scales = a_scales;
  p.w_scales = w_scales;
  p.C = C;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.status = status;
  CUtensorMap tw, tx;
  int r = make_tensormap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, W, N, K, ldw, BW, SLAB, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  r = make_tensormap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, A, M, K, lda, p.box, SLAB, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  int grid = p.num_n_tiles * p.splits;
  if (p.splits == 1) {
    const int most = max_ctas > 0 ? max_ctas : 2 * sm_count();
    if (grid > most) grid = most;
    return p.tn == 32 ? launch_fp8_stream<32, false, false>(tw, tx, p, grid, stream)
                      : launch_fp8_stream<64, false, false>(tw, tx, p, grid, stream);
  }
  return p.tn == 32 ? launch_fp8_stream<32, false, true>(tw, tx, p, grid, stream)
                    : launch_fp8_stream<64, false, true>(tw, tx, p, grid, stream);
}

// The operands of b200_grouped_gemm_fp8_block.
extern "C" int b200_grouped_gemm_fp8_stream(const void* A, const float* a_scales, const void* W, const float* w_scales,
                                            void* C, const int* expert_offsets, int num_experts, int total_rows, int N,
                                            int K, int lda, int ldc, int scale_rows, int swiglu, int up_scale_row0,
                                            int* status, int max_ctas, cudaStream_t stream) {
  using namespace fp8s;
  if (total_rows <= 0 || num_experts <= 0 || N <= 0 || K <= 0) return 0;
  if (num_experts > MAX_EXPERTS) return -13;
  if ((K % SLAB) != 0) return -10;
  if (swiglu && (N % 16) != 0) return -11;
  Fp8StreamParams p{};
  p.M = total_rows;
  p.N = N;
  p.k_slabs = K / SLAB;
  p.tn = MAX_ROWS;
  p.box = 16;
  p.stages = RING / (W_BYTES + p.tn * SLAB);
  p.num_n_tiles = (N + BW - 1) / BW;
  p.splits = 1;
  p.num_experts = num_experts;
  p.scale_rows = scale_rows;
  p.up_scale_row0 = up_scale_row0;
  p.ldc = ldc;
  p.swiglu = swiglu;
  p.a_scales = a_scales;
  p.w_scales = w_scales;
  p.C = C;
  p.expert_offsets = expert_offsets;
  p.status = status;
  const long long row_tiles = total_rows / p.tn + (num_experts < total_rows ? num_experts : total_rows);
  if (row_tiles * p.num_n_tiles > 0x3fffffffll) return -14;
  CUtensorMap tw, tx;
  int r = make_tensormap_3d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, W, num_experts, N, K, static_cast<uint64_t>(N) * K, K, BW,
                            SLAB, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  r = make_tensormap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, A, total_rows, K, lda, p.box, SLAB,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  int grid = max_ctas > 0 ? max_ctas : 2 * sm_count();
  if (row_tiles * p.num_n_tiles < grid) grid = static_cast<int>(row_tiles * p.num_n_tiles);
  return launch_fp8_stream<64, true, false>(tw, tx, p, grid, stream);
}
