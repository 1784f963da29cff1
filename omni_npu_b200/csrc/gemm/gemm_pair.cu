// Products with many rows on CTA pairs, dense and grouped:  C[M,N] = A[M,K] * W[N,K]^T, bf16 / e4m3 in, fp32 accumulate.
// Two CTAs of a cluster (the two SMs of a TPC) compute one tile with tcgen05.mma.cta_group::2.
//
// The weights are the M operand (256 rows of W per tile, 128 in each CTA) and the rows of A the N operand, at most 256 per
// tile in steps of 32.  Each CTA stages its 128 rows of W and half of the tile's rows of A.
//   Grouped: an expert's rows are dealt out evenly to its tiles, so that a product spends no time on the rest of a 128-
//   or 256-row block that an expert does not fill (a quarter of the work at 512 rows per expert in blocks of 256).
//   Dense: the host picks the width that leaves the pairs the least idle time in their last wave (pair_width).
//
// Measured (us, 128- or 256-row blocks of A as the M operand / here / at the measured matrix rate): 128 experts, 512 rows
// each, 1536 x 2048 with silu 510 / 351 / 255, 2048 x 768 316 / 212 / 127 (there the 370 MB of results and rows weigh half
// as much again); 64 experts, 768 rows each, 2816 x 2048 652 / 435 / 350.
// Dense: 5632 x 2048 with silu 100 rows 17.2 / 12.8 / 3.6, 512 rows 24.6 / 16.7 / 7.3, 1024 rows 42.5 / 28.6 / 14.6;
// 28672 x 4096 with silu 512 rows 134 / 97 / 74, 8192 rows 1350 / 1280 / 1189; 4096 x 4096 400 rows 25.4 / 20.6 / 8.3.
// Copies of 32 rows of A instead of one or two took 495 for the third: the thread that starts the copies was late.
//
// What bounds it: what an SM takes in from L2 (some 85 GB/s, 0.74 us for the 64 KB of a full stage, which the tensor cores
// work off in 0.55), in long runs the power limit.  Per CTA (320 threads): warp 0 TMA,
// warp 1 MMA (leader CTA only issues), warps 2-9 epilogue, four on each half of the tile's rows; two accumulators, so
// that the epilogue of a tile runs under the products of the next.  A thread of the epilogue holds one column of C
// (column_store.cuh).
//
// Barriers: full[s] and tmem_empty[a] in the leader (bytes and arrivals of both CTAs), empty[s] and tmem_full[a] in both
// (one commit arrives at the two).  Plain per-CTA loads, no multicast.  CTA-scope try_wait: the cluster-scope acquire form
// costs some 300 clocks a call even on a completed barrier.  Every wait is bounded; on expiry the pair records a status
// code, waits for what is in flight, frees its TMEM and returns.

#include "../common/device_once.h"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "column_store.cuh"
#include "group_tiles.cuh"

namespace b200 {

namespace pair {
constexpr int BW = 256;                  // rows of W per tile of a pair
constexpr int MAX_ROWS = 256;            // rows of A per tile
constexpr int BOX = 32;                  // rows of A that a CTA stages: 32, 64, 96 or 128, in one or two copies
constexpr int KSUB = 2;                  // 128-byte slabs of K per stage: fewer barrier round trips
constexpr int SLAB = 128 * 128;          // 128 rows x 128 bytes
constexpr int RING = 216 * 1024;
constexpr int THREADS = 320;
constexpr int MAX_EXPERTS = 512;
}  // namespace pair

struct PairParams {
  int M, N, k_iters, num_n_tiles, num_experts, ldc, out_fp32, act;
  int slab_elems;          // elements of K in 128 bytes
  int width;               // dense: rows of A per tile
  int x_rows, stages;      // rows of A that a stage has room for, in each CTA; stages of the ring
  int w_ready;             // dense: no kernel still running writes W, its first ring goes ahead of the wait
  float act_alpha, act_limit;
  void* C;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  const int* expert_offsets;
  int* status;
};

struct PairTile {
  int n0, row0, rows, width, expert;
};

// Rows of A per tile of an expert with this many rows.
__device__ __forceinline__ int pair_group_width(int rows) {
  const int tiles = (rows + pair::MAX_ROWS - 1) / pair::MAX_ROWS;
  return tiles ? ((rows + tiles - 1) / tiles + 31) & ~31 : 32;
}

template <bool GROUPED>
__device__ __forceinline__ bool pair_tile(const PairParams& p, const int* prefix, const int* first_row, int t, int& cursor,
                                          PairTile& tile) {
  if constexpr (GROUPED) {
    if (t >= prefix[p.num_experts]) return false;
    while (prefix[cursor + 1] <= t) ++cursor;
    const int row0 = first_row[cursor], rows = first_row[cursor + 1] - row0;
    const int w = pair_group_width(rows);
    const int row_tiles = (rows + w - 1) / w;
    const int local = t - prefix[cursor], rt = local % row_tiles;
    tile.n0 = local / row_tiles * pair::BW;
    tile.row0 = row0 + rt * w;
    tile.rows = min(w, rows - rt * w);
    tile.expert = cursor;
  } else {
    const int row_tiles = (p.M + p.width - 1) / p.width;
    const int nt = t / row_tiles, rt = t - nt * row_tiles;
    if (nt >= p.num_n_tiles) return false;
    tile.n0 = nt * pair::BW;
    tile.row0 = rt * p.width;
    tile.rows = min(p.width, p.M - tile.row0);
    tile.expert = 0;
  }
  tile.width = (tile.rows + 31) & ~31;
  return true;
}

template <bool GROUPED, bool FP8>
__global__ void __launch_bounds__(pair::THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                    const __grid_constant__ CUtensorMap tm_x64, const __grid_constant__ CUtensorMap tm_x32,
                    const PairParams p) {
  using namespace pair;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int x_slab = p.x_rows * 128, stage_bytes = KSUB * (SLAB + x_slab);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty_bar = full_bar + p.stages;
  uint64_t* tmem_full = empty_bar + p.stages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* drain_bar = tmem_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* prefix = const_cast<int*>(abort_flag) + 1;       // grouped: tiles before an expert, [E + 1]
  int* first_row = prefix + p.num_experts + 1;          // the offsets

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 16);       // 8 epilogue warps of each CTA
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_x64);
    tma_prefetch_desc(&tm_x32);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  if constexpr (GROUPED) {
    pdl_wait();      // the offsets come from an earlier kernel
    if (warp == 2)
      group_tiles(p.expert_offsets, p.num_experts, prefix, first_row, [&](int rows) {
        const int w = pair_group_width(rows);
        return (rows + w - 1) / w * p.num_n_tiles;
      });
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();          // both CTAs' barriers exist before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int t_first = blockIdx.x >> 1, t_stride = gridDim.x >> 1;
  pdl_trigger();
  // weights that no kernel ahead of this one writes (the caller says so): their first ring is under way before the wait
  const bool early = !GROUPED && p.w_ready && threadIdx.x == 0;
  if (!early) pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0, cursor = 0, preloaded = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      PairTile tile;
      // the leader's barrier collects the bytes of both CTAs
      const auto expect = [&](int s) {
        const int staged = (tile.width / 2 + BOX - 1) & ~(BOX - 1);
        if (leader) mbar_arrive_expect_tx(&full_bar[s], static_cast<uint32_t>(2 * KSUB * (SLAB + staged * 128)));
      };
      const auto load_w = [&](int s, int k) {
        const uint32_t bar = mapa_shared(smem_u32(&full_bar[s]), 0);
#pragma unroll
        for (int j = 0; j < KSUB; ++j) {
          uint8_t* dst = smem + s * stage_bytes + j * SLAB;
          if constexpr (GROUPED)
            tma_load_3d_pair(dst, &tm_w, bar, (k * KSUB + j) * p.slab_elems, tile.n0 + rank * 128, tile.expert);
          else
            tma_load_2d_pair(dst, &tm_w, bar, (k * KSUB + j) * p.slab_elems, tile.n0 + rank * 128);
        }
      };
      if (early) {
        if (pair_tile<GROUPED>(p, prefix, first_row, t_first, cursor, tile))
          for (; preloaded < p.stages && preloaded < p.k_iters; ++preloaded) {
            expect(preloaded);
            load_w(preloaded, preloaded);
          }
        pdl_wait();
      }
      for (int t = t_first; ok && pair_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        const int half = tile.width / 2, staged = (half + BOX - 1) & ~(BOX - 1);
        const int row = tile.row0 + rank * half;
        for (int k = 0; k < p.k_iters; ++k) {
          if (issued >= preloaded) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
              atomicCAS(p.status, 0, kStatusTimeoutEmptyBarrier);
              *abort_flag = 1;
              ok = false;
              break;
            }
            expect(stage);
            load_w(stage, k);
          }
          const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0);
#pragma unroll
          for (int j = 0; j < KSUB; ++j) {
            const int kc = (k * KSUB + j) * p.slab_elems;
            uint8_t* x = smem + stage * stage_bytes + KSUB * SLAB + j * x_slab;
            if (staged == 128) tma_load_2d_pair(x, &tm_x, bar, kc, row);
            if (staged == 64 || staged == 96) tma_load_2d_pair(x, &tm_x64, bar, kc, row);
            if (staged == 32 || staged == 96)
              tma_load_2d_pair(x + (staged - BOX) * 128, &tm_x32, bar, kc, row + staged - BOX);
          }
          ++issued;
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok && leader) {
        // wait, bounded, until the copies of both CTAs have landed (the peer meets this CTA at the end)
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
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (leader && lane == 0) {
      int stage = 0, cursor = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      PairTile tile;
      const uint32_t lo0 = (smem_u32(smem) & 0x3FFFF) >> 4;
      for (int t = t_first; ok && pair_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        if (*abort_flag || !mbar_wait(&tmem_empty[acc], acc_phase ^ 1)) {
          if (!*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemEmpty);
          *abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t idesc = make_idesc(FP8 ? 0 : 1, FP8 ? 0 : 1, BW, tile.width);
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * 256);
        for (int k = 0; k < p.k_iters; ++k) {
          if (!mbar_wait(&full_bar[stage], phase)) {
            atomicCAS(p.status, 0, kStatusTimeoutFullBarrier);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          uint32_t w_lo = lo0 + ((stage * stage_bytes) >> 4), x_lo = w_lo + ((KSUB * SLAB) >> 4);
#pragma unroll
          for (int j = 0; j < KSUB; ++j, w_lo += SLAB >> 4, x_lo += x_slab >> 4) {
            umma_pair_first<FP8>(d, w_lo, x_lo, idesc, (k > 0 || j > 0) ? 1u : 0u);
            umma_pair_acc<FP8>(d, w_lo + 2, x_lo + 2, idesc);
            umma_pair_acc<FP8>(d, w_lo + 4, x_lo + 4, idesc);
            umma_pair_acc<FP8>(d, w_lo + 6, x_lo + 6, idesc);
          }
          // the stage is free in both CTAs once these MMAs retire
          tc_commit_pair_both(smem_u32(&empty_bar[stage]));
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit_pair_both(smem_u32(&tmem_full[acc]));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int quarter = warp & 3, part = (warp - 2) >> 2;       // TMEM lanes; half of the rows
    // bf16 results without a residual, and without a bias behind a unary activation, are stored in pairs of columns
    const bool plain = act_is_gated(p.act) || (!p.out_fp32 && !p.residual && !(p.bias && act_is_unary(p.act)));
    const bool pairs = columns_pair(p.C, p.ldc, p.N, act_is_gated(p.act));
    const bool plain32 = !GROUPED && p.out_fp32 && !p.residual && p.act == kActNone;
    int cursor = 0, acc = 0;
    uint32_t acc_phase = 0;
    PairTile tile;
    for (int t = t_first; pair_tile<GROUPED>(p, prefix, first_row, t, cursor, tile); t += t_stride) {
      bool ok = !*abort_flag && mbar_wait(&tmem_full[acc], acc_phase);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0 && !*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemFull);
        *abort_flag = 1;
        break;
      }
      tc_fence_after_sync();
      const uint32_t col = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * 256);
      const int n = tile.n0 + rank * 128 + quarter * 32 + lane;
      const int mid = tile.width / 2;       // a multiple of 16
      const int c_end = part ? tile.rows : min(mid, tile.rows);
      const float bias = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
      for (int c = part ? mid : 0; c < c_end; c += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(col + static_cast<uint32_t>(c))
            : "memory");
        tmem_ld_wait();
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[i]);
        const size_t at = static_cast<size_t>(tile.row0 + c) * p.ldc;
        const int rows = tile.rows - c;
        if (plain) {
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] += bias;
          store_act_columns(p.act, p.act_alpha, p.act_limit, x, static_cast<__nv_bfloat16*>(p.C) + at, p.ldc, n, p.N, rows,
                            pairs);
        } else if (plain32) {
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] += bias;
          store_fp32_columns(x, static_cast<float*>(p.C) + at, p.ldc, n, p.N, rows);
        } else if (n < p.N) {
          float add[16];
#pragma unroll
          for (int i = 0; i < 16; ++i)
            add[i] = p.residual && i < rows ? __bfloat162float(p.residual[at + static_cast<size_t>(i) * p.ldc + n]) : 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (act_is_unary(p.act)) x[i] = unary_act(p.act, x[i], p.act_alpha, p.act_limit);
            x[i] += bias;
            x[i] += add[i];
            if (i >= rows) continue;
            if (p.out_fp32)
              static_cast<float*>(p.C)[at + static_cast<size_t>(i) * p.ldc + n] = x[i];
            else
              static_cast<__nv_bfloat16*>(p.C)[at + static_cast<size_t>(i) * p.ldc + n] = __float2bfloat16(x[i]);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tmem_empty[acc]), 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  // ------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (leader && warp == 1 && lane == 0 && *abort_flag) {
    tc_commit_pair(smem_u32(drain_bar));
    mbar_wait(drain_bar, 0);
  }
  // neither CTA may retire (or free TMEM) while its peer can still signal it or the leader's MMAs can still write it
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Rows of A per tile of a dense product: the width at which the pairs' waves cost least, a tile of w rows taking time in
// proportion to the w + 256 rows that it loads (28672 x 4096: 22.4 us a wave with 224, 19.6 with 160).  400 rows of that
// product take 90 us in 4 waves of 224 and 98 in 5 of 160; 1023 rows of 6144 x 4096 44 in 2 of 192 and 47 in 2 of 256.
static int pair_width(int M, int n_tiles, int pairs) {
  int best = pair::MAX_ROWS;
  long long best_cost = -1;
  for (int w = pair::MAX_ROWS; w >= 32; w -= 32) {
    const long long tiles = static_cast<long long>(n_tiles) * ((M + w - 1) / w);
    const long long cost = (tiles + pairs - 1) / pairs * (w + 256);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = w;
    }
  }
  return best;
}

template <bool GROUPED, bool FP8>
static int launch_pair(const void* A, const void* W, int rows, int K, int lda, int ldw, PairParams& p, long long most,
                       int max_ctas, cudaStream_t stream) {
  using namespace pair;
  constexpr int eb = FP8 ? 1 : 2;
  constexpr CUtensorMapDataType dt = FP8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  p.slab_elems = 128 / eb;
  p.k_iters = (K + KSUB * p.slab_elems - 1) / (KSUB * p.slab_elems);
  p.stages = RING / (KSUB * (SLAB + p.x_rows * 128));
  if (p.stages > 6) p.stages = 6;
  CUtensorMap tw, tx[3];
  int r = GROUPED ? make_tensormap_3d(&tw, dt, eb, W, p.num_experts, p.N, K, static_cast<uint64_t>(p.N) * K, K, 128,
                                      p.slab_elems, CU_TENSOR_MAP_SWIZZLE_128B)
                  : make_tensormap_2d(&tw, dt, eb, W, p.N, K, ldw, 128, p.slab_elems, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  for (int i = 0; i < 3; ++i) {
    r = make_tensormap_2d(&tx[i], dt, eb, A, rows, K, lda, 128 >> i, p.slab_elems, CU_TENSOR_MAP_SWIZZLE_128B);
    if (r) return r - 1000;
  }
  auto kern = gemm_pair_kernel<GROUPED, FP8>;
  static DeviceOnce once;
  int dev = 0;
  if (once.needed(&dev)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return -20;
    once.mark(dev);
  }
  const long long pairs = most < max_ctas / 2 ? most : max_ctas / 2;
  const size_t smem = 1024 + p.stages * KSUB * (SLAB + p.x_rows * 128) + (2 * p.stages + 5) * 8 + 8 +
                      (GROUPED ? 2 * (p.num_experts + 1) * 4 : 0);
  return launch_pdl(kern, dim3(static_cast<unsigned>(2 * pairs)), dim3(THREADS), smem, stream, 2, tw, tx[0], tx[1], tx[2],
                    p) == cudaSuccess
             ? 0
             : -21;
}

static int pair_ctas(int max_ctas) {
  const int n = max_ctas > 0 && max_ctas < sm_count() ? max_ctas : sm_count();
  return n < 2 ? 2 : n;
}

}  // namespace b200

using namespace b200;

// Same contract as b200_gemm (no split-K).  width: rows of A per tile, a multiple of 32 up to 256; 0: by rule.
// w_ready: see PairParams.
extern "C" int b200_gemm_pair(const void* A, const void* W, void* C, const void* bias, const void* residual, int M, int N,
                              int K, int lda, int ldw, int ldc, int dtype_fp8, int out_fp32, int act, int width,
                              int* status, int max_ctas, float act_alpha, float act_limit, int w_ready, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (width != 0 && (width < 32 || width > 256 || (width % 32) != 0)) return -10;
  if (act_is_gated(act) && (N % 16) != 0) return -11;
  PairParams p{};
  const int ctas = pair_ctas(max_ctas);
  p.M = M;
  p.N = N;
  p.num_n_tiles = (N + pair::BW - 1) / pair::BW;
  p.width = width ? width : pair_width(M, p.num_n_tiles, ctas / 2);
  p.x_rows = (p.width / 2 + pair::BOX - 1) / pair::BOX * pair::BOX;
  p.ldc = ldc;
  p.out_fp32 = out_fp32;
  p.w_ready = w_ready;
  p.act = act;
  p.act_alpha = act_alpha;
  p.act_limit = act_limit;
  p.C = C;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.status = status;
  const long long tiles = static_cast<long long>(p.num_n_tiles) * ((M + p.width - 1) / p.width);
  if (tiles > 0x3fffffffll) return -14;
  return dtype_fp8 ? launch_pair<false, true>(A, W, M, K, lda, ldw, p, tiles, ctas, stream)
                   : launch_pair<false, false>(A, W, M, K, lda, ldw, p, tiles, ctas, stream);
}

// A [total_rows, K] (pitch lda), W [E, N, K], C [total_rows, N, or N / 2 with a gated activation]; rows
// expert_offsets[e] .. expert_offsets[e + 1] (device) belong to expert e.
extern "C" int b200_grouped_gemm_pair(const void* A, const void* W, void* C, const int* expert_offsets, int num_experts,
                                      int total_rows, int N, int K, int lda, int ldc, int act, int* status, int max_ctas,
                                      float act_alpha, float act_limit, cudaStream_t stream) {
  if (total_rows <= 0 || num_experts <= 0 || N <= 0 || K <= 0) return 0;
  if (num_experts > pair::MAX_EXPERTS) return -13;
  if (act_is_gated(act) && (N % 16) != 0) return -11;
  PairParams p{};
  p.N = N;
  p.num_n_tiles = (N + pair::BW - 1) / pair::BW;
  p.x_rows = pair::MAX_ROWS / 2;
  p.num_experts = num_experts;
  p.ldc = ldc;
  p.act = act;
  p.act_alpha = act_alpha;
  p.act_limit = act_limit;
  p.C = C;
  p.expert_offsets = expert_offsets;
  p.status = status;
  // a tile that is not an expert's last has more than 128 rows
  const long long most = (static_cast<long long>(total_rows) / 128 + num_experts) * p.num_n_tiles;
  if (most > 0x3fffffffll) return -14;
  return launch_pair<true, false>(A, W, total_rows, K, lda, K, p, most, pair_ctas(max_ctas), stream);
}
