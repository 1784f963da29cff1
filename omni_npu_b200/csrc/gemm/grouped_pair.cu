// Grouped products with many rows per expert on CTA pairs:  C[rows of e, N] = A[rows of e, K] * W[e][N, K]^T, bf16 in,
// fp32 accumulate.  Two CTAs of a cluster (the two SMs of a TPC) compute one tile with tcgen05.mma.cta_group::2.
//
// The weights are the M operand (256 rows of W per tile, 128 in each CTA) and the rows of A the N operand: an expert's
// rows are dealt out evenly to tiles of at most 256, each a multiple of 32 wide, so that a product spends no time on the
// rest of a 128- or 256-row block that an expert does not fill (a quarter of the work at 512 rows per expert in blocks
// of 256).  Each CTA stages its 128 rows of W and half of the tile's rows of A.
//
// Measured (us, gemm_tcgen05_kernel / here / at the measured matrix rate): 128 experts, 512 rows each, 1536 x 2048 with
// silu 510 / 351 / 255, 2048 x 768 316 / 212 / 127 (there the 370 MB of results and rows weigh half as much again); 64
// experts, 768 rows each, 2816 x 2048 652 / 435 / 350.  Copies of 32 rows of A instead of one or two took 495 for the last:
// the thread that starts the copies was late.
//
// What bounds it: the tensor cores.  Per CTA (320 threads): warp 0 TMA, warp 1 MMA (leader CTA only issues), warps 2-9
// epilogue, four on each half of the tile's rows; two accumulators, so that the epilogue of a tile runs under the
// products of the next.  A thread of the epilogue holds one column of C (column_store.cuh).
//
// Barriers as in gemm_pair_kernel: full[s] and tmem_empty[a] in the leader, empty[s] and tmem_full[a] in both.  Plain
// per-CTA loads, no multicast.  Every wait is bounded; on expiry the pair records a status code, waits for what is in
// flight, frees its TMEM and returns.

#include "../common/device_once.h"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "column_store.cuh"

namespace b200 {

namespace gpair {
constexpr int BW = 256;                  // rows of W per tile of a pair
constexpr int MAX_ROWS = 256;            // rows of A per tile
constexpr int BOX = 32;                  // rows of A that a CTA stages: 32, 64, 96 or 128, in one or two copies
constexpr int KSUB = 2;                  // 128-byte slabs of K per stage
constexpr int STAGES = 3;
constexpr int SLAB = 128 * 128;          // 128 rows x 128 bytes
constexpr int W_BYTES = KSUB * SLAB, STAGE_BYTES = 2 * W_BYTES;
constexpr int THREADS = 320;
constexpr int MAX_EXPERTS = 512;
}  // namespace gpair

struct GroupedPairParams {
  int N, k_iters, num_n_tiles, num_experts, ldc, act;
  float act_alpha, act_limit;
  __nv_bfloat16* C;
  const int* expert_offsets;
  int* status;
};

struct GroupedPairTile {
  int n0, row0, rows, width, expert;
};

// Rows of A per tile of an expert with this many rows.
__device__ __forceinline__ int gpair_width(int rows) {
  const int tiles = (rows + gpair::MAX_ROWS - 1) / gpair::MAX_ROWS;
  return tiles ? ((rows + tiles - 1) / tiles + 31) & ~31 : 32;
}

__device__ __forceinline__ bool gpair_tile(const GroupedPairParams& p, const int* prefix, const int* first_row, int t,
                                           int& cursor, GroupedPairTile& tile) {
  if (t >= prefix[p.num_experts]) return false;
  while (prefix[cursor + 1] <= t) ++cursor;
  const int row0 = first_row[cursor], rows = first_row[cursor + 1] - row0;
  const int w = gpair_width(rows);
  const int row_tiles = (rows + w - 1) / w;
  const int local = t - prefix[cursor], rt = local % row_tiles;
  tile.n0 = local / row_tiles * gpair::BW;
  tile.row0 = row0 + rt * w;
  tile.rows = min(w, rows - rt * w);
  tile.width = (tile.rows + 31) & ~31;
  tile.expert = cursor;
  return true;
}

__global__ void __launch_bounds__(gpair::THREADS, 1)
grouped_pair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                    const __grid_constant__ CUtensorMap tm_x64, const __grid_constant__ CUtensorMap tm_x32,
                    const GroupedPairParams p) {
  using namespace gpair;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* drain_bar = tmem_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* prefix = const_cast<int*>(abort_flag) + 1;       // tiles before an expert, [E + 1]
  int* first_row = prefix + p.num_experts + 1;          // the offsets

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
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
  pdl_wait();
  if (warp == 2) {
    const int per = (p.num_experts + 31) / 32;
    const int e0 = min(p.num_experts, lane * per), e1 = min(p.num_experts, e0 + per);
    const auto tiles_of = [&](int rows) {
      const int w = gpair_width(rows);
      return (rows + w - 1) / w * p.num_n_tiles;
    };
    int tiles = 0;
    for (int e = e0; e < e1; ++e) tiles += tiles_of(p.expert_offsets[e + 1] - p.expert_offsets[e]);
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int before = incl - tiles;
    for (int e = e0; e < e1; ++e) {
      const int a = p.expert_offsets[e], b = p.expert_offsets[e + 1];
      prefix[e] = before;
      first_row[e] = a;
      before += tiles_of(b - a);
      if (e + 1 == p.num_experts) {
        prefix[e + 1] = before;
        first_row[e + 1] = b;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();          // both CTAs' barriers exist before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int t_first = blockIdx.x >> 1, t_stride = gridDim.x >> 1;
  pdl_trigger();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0, cursor = 0;
      uint32_t phase = 0, issued = 0;
      bool ok = true;
      GroupedPairTile tile;
      for (int t = t_first; ok && gpair_tile(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        const int half = tile.width / 2, staged = (half + BOX - 1) & ~(BOX - 1);
        const int row = tile.row0 + rank * half;
        for (int k = 0; k < p.k_iters; ++k) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            atomicCAS(p.status, 0, kStatusTimeoutEmptyBarrier);
            *abort_flag = 1;
            ok = false;
            break;
          }
          // the leader's barrier collects the bytes of both CTAs
          if (leader)
            mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>(2 * KSUB * (SLAB + staged * 128)));
          const uint32_t full_leader = mapa_shared(smem_u32(&full_bar[stage]), 0);
          uint8_t* dst = smem + stage * STAGE_BYTES;
          for (int j = 0; j < KSUB; ++j) {
            const int kc = (k * KSUB + j) * 64;
            tma_load_3d_pair(dst + j * SLAB, &tm_w, full_leader, kc, tile.n0 + rank * 128, tile.expert);
            uint8_t* x = dst + W_BYTES + j * SLAB;
            if (staged == 128) tma_load_2d_pair(x, &tm_x, full_leader, kc, row);
            if (staged == 64 || staged == 96) tma_load_2d_pair(x, &tm_x64, full_leader, kc, row);
            if (staged == 32 || staged == 96)
              tma_load_2d_pair(x + (staged - BOX) * 128, &tm_x32, full_leader, kc, row + staged - BOX);
          }
          ++issued;
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok && leader) {
        // wait, bounded, until the copies of both CTAs have landed (the peer meets this CTA at the end)
        for (uint32_t i = 0; i < STAGES && i < issued; ++i) {
          if (--stage < 0) {
            stage = STAGES - 1;
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
      GroupedPairTile tile;
      const uint32_t lo0 = (smem_u32(smem) & 0x3FFFF) >> 4;
      for (int t = t_first; ok && gpair_tile(p, prefix, first_row, t, cursor, tile); t += t_stride) {
        if (*abort_flag || !mbar_wait(&tmem_empty[acc], acc_phase ^ 1)) {
          if (!*abort_flag) atomicCAS(p.status, 0, kStatusTimeoutTmemEmpty);
          *abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t idesc = make_idesc(1, 1, BW, tile.width);
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * 256);
        for (int k = 0; k < p.k_iters; ++k) {
          if (!mbar_wait(&full_bar[stage], phase)) {
            atomicCAS(p.status, 0, kStatusTimeoutFullBarrier);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          uint32_t w_lo = lo0 + ((stage * STAGE_BYTES) >> 4), x_lo = w_lo + (W_BYTES >> 4);
#pragma unroll
          for (int j = 0; j < KSUB; ++j, w_lo += SLAB >> 4, x_lo += SLAB >> 4) {
            umma_pair_first<false>(d, w_lo, x_lo, idesc, (k > 0 || j > 0) ? 1u : 0u);
            umma_pair_acc<false>(d, w_lo + 2, x_lo + 2, idesc);
            umma_pair_acc<false>(d, w_lo + 4, x_lo + 4, idesc);
            umma_pair_acc<false>(d, w_lo + 6, x_lo + 6, idesc);
          }
          // the stage is free in both CTAs once these MMAs retire
          tc_commit_pair_both(smem_u32(&empty_bar[stage]));
          if (++stage == STAGES) {
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
    const bool pairs = columns_pair(p.C, p.ldc, p.N, act_is_gated(p.act));
    int cursor = 0, acc = 0;
    uint32_t acc_phase = 0;
    GroupedPairTile tile;
    for (int t = t_first; gpair_tile(p, prefix, first_row, t, cursor, tile); t += t_stride) {
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
      __nv_bfloat16* out = p.C + static_cast<size_t>(tile.row0) * p.ldc;
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
        store_act_columns(p.act, p.act_alpha, p.act_limit, x, out + static_cast<size_t>(c) * p.ldc, p.ldc, n, p.N,
                          tile.rows - c, pairs);
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

}  // namespace b200

using namespace b200;

// A [total_rows, K] (pitch lda), W [E, N, K], C [total_rows, N, or N / 2 with a gated activation]; rows
// expert_offsets[e] .. expert_offsets[e + 1] (device) belong to expert e.
extern "C" int b200_grouped_gemm_pair(const void* A, const void* W, void* C, const int* expert_offsets, int num_experts,
                                      int total_rows, int N, int K, int lda, int ldc, int act, int* status, int max_ctas,
                                      float act_alpha, float act_limit, cudaStream_t stream) {
  using namespace gpair;
  if (total_rows <= 0 || num_experts <= 0 || N <= 0 || K <= 0) return 0;
  if (num_experts > MAX_EXPERTS) return -13;
  if (act_is_gated(act) && (N % 16) != 0) return -11;
  GroupedPairParams p{};
  p.N = N;
  p.k_iters = (K + KSUB * 64 - 1) / (KSUB * 64);
  p.num_n_tiles = (N + BW - 1) / BW;
  p.num_experts = num_experts;
  p.ldc = ldc;
  p.act = act;
  p.act_alpha = act_alpha;
  p.act_limit = act_limit;
  p.C = static_cast<__nv_bfloat16*>(C);
  p.expert_offsets = expert_offsets;
  p.status = status;
  // a tile that is not an expert's last has more than 128 rows
  const long long most = (static_cast<long long>(total_rows) / 128 + num_experts) * p.num_n_tiles;
  if (most > 0x7fffffffll) return -14;
  CUtensorMap tw, tx[3];
  int r = make_tensormap_3d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, num_experts, N, K, static_cast<uint64_t>(N) * K,
                            K, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r;
  for (int i = 0; i < 3; ++i) {
    r = make_tensormap_2d(&tx[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, total_rows, K, lda, 128 >> i, 64,
                          CU_TENSOR_MAP_SWIZZLE_128B);
    if (r) return r - 1000;
  }
  static DeviceOnce once;
  int dev = 0;
  if (once.needed(&dev)) {
    if (cudaFuncSetAttribute(grouped_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
      return -20;
    once.mark(dev);
  }
  int pairs = (max_ctas > 0 && max_ctas < sm_count() ? max_ctas : sm_count()) / 2;
  if (pairs < 1) pairs = 1;
  if (most < pairs) pairs = static_cast<int>(most);
  const size_t smem = 1024 + STAGES * STAGE_BYTES + (2 * STAGES + 5) * 8 + 8 + 2 * (num_experts + 1) * 4;
  return launch_pdl(grouped_pair_kernel, dim3(2 * pairs), dim3(THREADS), smem, stream, 2, tw, tx[0], tx[1], tx[2],
                    p) == cudaSuccess
             ? 0
             : -21;
}
