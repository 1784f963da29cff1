// Paged GQA prefill attention on the 5th-generation tensor cores: query / key head size 128 or 192 (non-absorbed
// latent attention: 128 + 64 rotated), value head size 128, bf16.
//
// A CTA works on two tiles of 128 query rows at once: the same rows of two query heads that share a key / value head
// (an even number of heads per key / value head), else two neighbouring row tiles of one head.  The two tiles take turns: while the softmax of one runs, the
// tensor cores multiply for the other.  Per key tile of 128 keys and query tile
//   S = Q K^T   M = 128, N = 128, K = 128 or 192, operands in shared memory (K straight from the paged cache by TMA),
//               accumulator in TMEM;
//   P = exp2(S - max) written back over S as bf16: the A operand of the second product lies in TMEM, so that P never
//               passes through shared memory;
//   O += P V    M = 128, N = 128, K = 128 keys; V as it lies in the cache, through an MN-major descriptor.
// TMEM: S0 | S1 | O0 | O1, 128 columns each.  A row of a tile belongs to one thread (tcgen05.ld gives a thread its
// row): no shuffles.  The reference maximum moves only when it is exceeded by 2^8, which keeps the rescale of O rare.
//
// What bounds it: exp2.  A key tile costs 2 x 128 x 128 of them, 2048 clocks of an SM's special function units, and
// its four products 2048 clocks of the tensor core; the two overlap.  The earlier form (one tile of 128 x 64 per CTA,
// two CTAs per SM, P through shared memory) waited for that chain on every tile.
//
// Persistent: one CTA per SM walks the (row tile, sequence, head) items, late row tiles (most keys) first, so that the
// copies of the next item run under the end of this one.  Warps 0-3 and 4-7: softmax of tile 0 and 1; warp 8: TMA;
// warp 9: MMA issue; warps 10 and 11 only complete the warpgroup that gives registers away.
//
// FLAT (latent attention, 128 + 64 rotated): keys and values are rows of the up-projection [rows, heads x (128 key, 128
// value)] and the rotated part, shared by the heads, rows of the latents; a sequence's rows lie one after another, so that
// a tile is one copy per 64 columns, and nothing is repacked into per-head pages (4 x 2048 tokens of 16 heads: the copies
// that did took 250 us a layer, the attention 151, and 119 in this form).
//
// Every wait is bounded; on expiry the CTA records a status code, stops issuing, waits for what is in flight, frees its
// TMEM and returns (its output rows are then not valid).
//
// Replaces npu_fused_infer_attention_score in its TND paged prefill form
// (omni_npu/attention/backends/attention.py:216-281).

#include "attn_params.cuh"
#include "../common/device_once.h"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "umma_desc.cuh"

namespace b200 {

namespace two {
constexpr int BM = 128;                 // query rows of a tile
constexpr int BN = 128;                 // keys per tile
constexpr int DV = 128;
constexpr int THREADS = 384;
// registers: a thread of the softmax holds its row of S; the two warps that issue need few.  The shares must fit what
// the launch takes (THREADS x MIN_REGS), or setmaxnreg would wait for good: checked before the first launch (a compiler
// that gives the kernel fewer makes the callers take their other kernels).
constexpr int SOFTMAX_REGS = 208, ISSUE_REGS = 56, MIN_REGS = 160;
static_assert(256 * SOFTMAX_REGS + 128 * ISSUE_REGS <= THREADS * MIN_REGS, "register split");
constexpr int SLAB = 128 * 128;         // 128 rows x 128 bytes
constexpr int V_BYTES = 2 * SLAB;
constexpr int COL_S = 0, COL_O = 256;   // of tile 0; tile 1 follows 128 columns later
constexpr int TMEM_COLS = 512;

template <int DQK>
struct Cfg {
  static constexpr int QK_SLABS = DQK / 64;
  static constexpr int Q_BYTES = QK_SLABS * SLAB;       // of one tile
  static constexpr int K_BYTES = QK_SLABS * SLAB;
  // a key tile is free as soon as both products with it are through, long before its values are: head size 192 has
  // room for one stage of keys
  static constexpr int KS = DQK == 128 ? 3 : 1, VS = 2;
  static constexpr int OFF_K = 2 * Q_BYTES;
  static constexpr int OFF_V = OFF_K + KS * K_BYTES;
  static constexpr int OFF_BAR = OFF_V + VS * V_BYTES;
  static constexpr int NUM_BARS = 2 + 2 * KS + 2 * VS + 6 + 1;
  static constexpr int SMEM = OFF_BAR + NUM_BARS * 8 + 16;
};
}  // namespace two

enum : int { kStatusPrefillTimeout = 41, kStatusPrefillSmemAlign = 42 };

// D[tmem] (+)= A[tmem] * B[smem], bf16
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

struct TwoTileItem {
  int h[2], m0[2], n[2];       // head, first row, key tiles of each query tile
  int n_max, b, q_begin, q_len, kv_len, ctx, kvh;
};

struct TwoTileGrid {
  int m_units, head_units, B, by_head, items;
};

__device__ __forceinline__ TwoTileItem two_tile_item(int idx, const TwoTileGrid& g, const AttnParams& p) {
  TwoTileItem it;
  const int hu = idx % g.head_units, rest = idx / g.head_units;
  it.b = rest % g.B;
  const int mu = g.m_units - 1 - rest / g.B;           // late rows see the most keys: first
  it.q_begin = p.cu_q[it.b];
  it.q_len = p.cu_q[it.b + 1] - it.q_begin;
  it.kv_len = p.seq_lens[it.b];
  it.ctx = it.kv_len - it.q_len;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    it.h[i] = g.by_head ? 2 * hu + i : hu;
    it.m0[i] = g.by_head ? mu * two::BM : (2 * mu + i) * two::BM;
    const int hi = p.causal ? min(it.kv_len, it.ctx + it.m0[i] + two::BM) : it.kv_len;
    it.n[i] = it.m0[i] < it.q_len ? (max(hi, 0) + two::BN - 1) / two::BN : 0;
  }
  it.n_max = max(it.n[0], it.n[1]);
  it.kvh = it.h[0] / (p.Hq / p.Hk);
  return it;
}

// FLAT: tm_k covers the up-projected rows, tm_v the rotated parts; block_tables[b] is sequence b's first row.
template <int DQK, bool FLAT>
__global__ void __launch_bounds__(two::THREADS, 1)
gqa_prefill_two_tiles_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                             const __grid_constant__ CUtensorMap tm_v, const AttnParams p, const int box_rows,
                             const TwoTileGrid g) {
  static_assert(!FLAT || DQK == 192, "latent attention");
  using namespace two;
  using C = Cfg<DQK>;
  constexpr int KS = C::KS, VS = C::VS;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;           // [KS]
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;          // [VS]
  uint64_t* v_empty = v_full + VS;
  uint64_t* s_full = v_empty + VS;          // [2], by query tile
  uint64_t* p_full = s_full + 2;
  uint64_t* o_done = p_full + 2;
  uint64_t* drain_bar = o_done + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((smem_u32(smem) & 1023u) != 0u) {      // the operand layouts need 1024-byte aligned slabs
    if (tid == 0 && p.status) atomicCAS(p.status, 0, kStatusPrefillSmemAlign);
    return;
  }
  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int s = 0; s < KS; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < VS; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  fence_proxy_async();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  pdl_trigger();
  pdl_wait();          // q and the cache rows of this step come from earlier kernels

  const auto give_up = [&]() {
    if (!*abort_flag && p.status) atomicCAS(p.status, 0, kStatusPrefillTimeout);
    *abort_flag = 1;
  };
  uint32_t q_loads = 0, k_loads = 0, v_loads = 0;      // copies started (producer warp)

  if (warp >= 8) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGS));
  if (warp == 8) {
    // ------------------------------------------------------------ TMA producer
    bool ok = true;
    for (int idx = blockIdx.x; ok && idx < g.items; idx += gridDim.x) {
      const TwoTileItem it = two_tile_item(idx, g, p);
      if (it.n_max == 0) continue;
      const int* bt = p.block_tables + static_cast<long long>(it.b) * p.max_blocks;
      const int first = FLAT ? bt[0] : 0;
      for (int j = 0; j < it.n_max; ++j) {
        const int n0 = j * BN;
        const int nboxes = FLAT ? 1 : (min(BN, it.kv_len - n0) + box_rows - 1) / box_rows;
        // keys (before the first tile's: the queries)
        if (j == 0) {
          if (q_loads > 0) ok = !*abort_flag && mbar_wait(q_empty, (q_loads - 1) & 1);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(q_full, C::Q_BYTES * ((it.n[0] > 0) + (it.n[1] > 0)));
            for (int i = 0; i < 2; ++i)
              if (it.n[i] > 0)
                for (int sl = 0; sl < C::QK_SLABS; ++sl)
                  tma_load_2d(smem + i * C::Q_BYTES + sl * SLAB, &tm_q, q_full, it.h[i] * DQK + sl * 64,
                              it.q_begin + it.m0[i]);
          }
          ++q_loads;
        }
        const int ks = static_cast<int>(k_loads % KS), vs = static_cast<int>(v_loads % VS);
        if (k_loads >= KS) ok = !*abort_flag && mbar_wait(&k_empty[ks], ((k_loads / KS) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&k_full[ks], static_cast<uint32_t>(nboxes * box_rows * 128) * C::QK_SLABS);
        __syncwarp();
        for (int l = lane; l < nboxes * C::QK_SLABS; l += 32) {
          if constexpr (FLAT) {
            // (keys past the sequence are masked, its values' rows cleared below; rows past the end read as zero)
            uint8_t* dst = smem + C::OFF_K + ks * C::K_BYTES + l * SLAB;
            if (l < 2)
              tma_load_2d(dst, &tm_k, &k_full[ks], it.h[0] * 256 + l * 64, first + n0);
            else
              tma_load_2d(dst, &tm_v, &k_full[ks], 0, first + n0);
            continue;
          }
          const int i = l / C::QK_SLABS, sl = l % C::QK_SLABS, key = n0 + i * box_rows;
          const int row = (bt[key / p.block_size] * p.Hk + it.kvh) * p.block_size + key % p.block_size;
          tma_load_2d(smem + C::OFF_K + ks * C::K_BYTES + sl * SLAB + i * box_rows * 128, &tm_k, &k_full[ks], sl * 64,
                      row);
        }
        ++k_loads;
        if (v_loads >= VS) ok = !*abort_flag && mbar_wait(&v_empty[vs], ((v_loads / VS) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&v_full[vs], static_cast<uint32_t>(nboxes * box_rows * 128) * 2);
        __syncwarp();
        for (int l = lane; l < nboxes * 2; l += 32) {
          if constexpr (FLAT) {
            tma_load_2d(smem + C::OFF_V + vs * V_BYTES + l * SLAB, &tm_k, &v_full[vs], it.h[0] * 256 + 128 + l * 64,
                        first + n0);
            continue;
          }
          const int i = l >> 1, sl = l & 1, key = n0 + i * box_rows;
          const int row = (bt[key / p.block_size] * p.Hk + it.kvh) * p.block_size + key % p.block_size;
          tma_load_2d(smem + C::OFF_V + vs * V_BYTES + sl * SLAB + i * box_rows * 128, &tm_v, &v_full[vs], sl * 64, row);
        }
        ++v_loads;
      }
    }
    if (!ok && lane == 0) give_up();
  } else if (warp == 9) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc(1, 1, BM, BN);                    // K-major A and B
      constexpr uint32_t idesc_o = make_idesc(1, 1, BM, DV) | (1u << 16);       // B (V) MN-major
      const uint32_t q_addr = smem_u32(smem), k_base = smem_u32(smem + C::OFF_K), v_base = smem_u32(smem + C::OFF_V);
      uint32_t items = 0, kc = 0, vc = 0, pc[2] = {0, 0};
      bool ok = true;
      const auto issue_qk = [&](int i, uint32_t k_addr) {
        // (descriptors count in 16 bytes; loops kept rolled: an unrolled one holds every descriptor in registers)
        uint64_t qd = make_smem_desc_sw128(q_addr + i * C::Q_BYTES), kd = make_smem_desc_sw128(k_addr);
#pragma unroll 1
        for (int slab = 0; slab < C::QK_SLABS; ++slab, qd += SLAB / 16, kd += SLAB / 16)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16(tmem_base + COL_S + i * 128, qd + kk * 2, kd + kk * 2, idesc_s, slab > 0 || kk > 0 ? 1u : 0u);
        tc_commit(&s_full[i]);
      };
      for (int idx = blockIdx.x; ok && idx < g.items; idx += gridDim.x) {
        const TwoTileItem it = two_tile_item(idx, g, p);
        if (it.n_max == 0) continue;
        ok = !*abort_flag && mbar_wait(q_full, items & 1) && mbar_wait(&k_full[kc % KS], (kc / KS) & 1);
        if (!ok) break;
        ++items;
        tc_fence_after_sync();
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (it.n[i] > 0) issue_qk(i, k_base + (kc % KS) * C::K_BYTES);
        tc_commit(&k_empty[kc % KS]);
        ++kc;
        if (it.n_max == 1) tc_commit(q_empty);
        for (int j = 0; j < it.n_max; ++j) {
          const bool more = j + 1 < it.n_max;
          ok = !*abort_flag && mbar_wait(&v_full[vc % VS], (vc / VS) & 1) &&
               (!more || mbar_wait(&k_full[kc % KS], (kc / KS) & 1));
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (j >= it.n[i]) continue;
            ok = mbar_wait(&p_full[i], pc[i] & 1);
            if (!ok) break;
            ++pc[i];
            tc_fence_after_sync();
            const uint64_t vd = desc_mnmajor(v_base + (vc % VS) * V_BYTES, SLAB);
            const int groups = (min(BN, it.kv_len - j * BN) + 15) / 16;
#pragma unroll 2
            for (int kk = 0; kk < groups; ++kk)        // 16 keys: 8 columns of P, 16 rows of 128 bytes of V
              umma_f16_ta(tmem_base + COL_O + i * 128, tmem_base + COL_S + i * 128 + kk * 8, vd + kk * 128, idesc_o,
                          (j > 0 || kk > 0) ? 1u : 0u);
            // in order behind the product that reads P: the next S may take its place
            if (j + 1 < it.n[i])
              issue_qk(i, k_base + (kc % KS) * C::K_BYTES);
            else
              tc_commit(&o_done[i]);
          }
          if (!ok) break;
          tc_commit(&v_empty[vc % VS]);
          ++vc;
          if (more) {
            tc_commit(&k_empty[kc % KS]);
            ++kc;
            if (j + 2 == it.n_max) tc_commit(q_empty);
          }
        }
      }
      if (!ok) give_up();
    }
  }
  } else {
    // ------------------------------------------------------------ softmax (one thread per row)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGS));
    const int t = warp >> 2;                              // query tile
    const int quarter = warp & 3;                         // TMEM lanes this warp may touch
    const int r = quarter * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_col = tmem_base + lanes + COL_S + t * 128, o_col = tmem_base + lanes + COL_O + t * 128;
    const float scale = p.scale_log2;
    uint32_t sc = 0, oc = 0, v_first = 0;                  // v_first: value tiles of the items before
    bool ok = true;
    for (int idx = blockIdx.x; ok && idx < g.items; idx += gridDim.x) {
      const TwoTileItem it = two_tile_item(idx, g, p);
      const int n = t ? it.n[1] : it.n[0], m0 = t ? it.m0[1] : it.m0[0], h = t ? it.h[1] : it.h[0];
      const uint32_t v_item = v_first;
      v_first += it.n_max;
      if (n == 0) {
        // rows that see no key: zero, of weight zero
        if (m0 + r < it.q_len) {
          const long long row = it.q_begin + m0 + r;
          uint4* dst = reinterpret_cast<uint4*>(p.out + row * p.out_stride + static_cast<long long>(h) * DV);
#pragma unroll
          for (int i = 0; i < DV / 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
          if (p.lse) p.lse[row * p.Hq + h] = -INFINITY;
        }
        continue;
      }
      const int row_lo = it.ctx + m0 + quarter * 32;      // smallest position in this warp
      const int limit = p.causal ? min(it.kv_len - 1, it.ctx + m0 + r) : it.kv_len - 1;    // last key this row sees
      float row_max = -INFINITY, row_sum = 0.f;
      for (int j = 0; j < n; ++j) {
        ok = !*abort_flag && mbar_wait(&s_full[t], sc & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ++sc;
        tc_fence_after_sync();
        uint32_t sv[4][32];
        const int n0 = j * BN;
        const bool whole = it.kv_len - n0 > BN / 2;           // else the second half of the tile's keys does not exist
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(s_col + c * 32, sv[c]);
        if (whole) {
          tmem_ld_32x32b_x32(s_col + 64, sv[2]);
          tmem_ld_32x32b_x32(s_col + 96, sv[3]);
        }
        tmem_ld_wait();
        // The second product reads whole groups of 16 keys.  Value rows past the sequence in the last one (the rest of a
        // page, another sequence's rows, what an earlier tile left) would count if they were infinite or NaN, although P
        // is zero there: the tile that the product comes first for clears them once they have landed.
        const int left = it.kv_len - n0;
        if (left < BN && (left & 15) != 0 && (t == 0 || j >= it.n[0])) {
          const uint32_t v = v_item + j;
          ok = __all_sync(0xffffffffu, mbar_wait(&v_full[v % VS], (v / VS) & 1));
          if (!ok) break;
          const int missing = 16 - (left & 15);
          for (int i = r; i < missing * 16; i += BM)
            *reinterpret_cast<uint4*>(smem + C::OFF_V + (v % VS) * V_BYTES + (i & 8 ? SLAB : 0) + (left + (i >> 4)) * 128 +
                                      (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          fence_proxy_async();
        }
        // tiles that lie entirely below the diagonal and inside the sequence need no mask
        if (!(n0 + BN <= it.kv_len && (!p.causal || n0 + BN - 1 <= row_lo))) {
          const int last = limit - n0;
#pragma unroll
          for (int c = 0; c < 128; ++c)
            if (c > last) sv[c >> 5][c & 31] = 0xff800000u;
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 32; ++c)
#pragma unroll
          for (int k = 0; k < 4; ++k) mx[k] = fmaxf(mx[k], __uint_as_float(sv[k][c]));
        const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale;
        // The reference maximum moves only when the tile's maximum exceeds it by more than 2^8: P then stays below
        // 256, the result is the same after the final division, and the rescale of O is rare.
        float new_max = row_max;
        if (tile_max > row_max + 8.f || row_max == -INFINITY) new_max = fmaxf(row_max, tile_max);
        const float corr = (new_max == -INFINITY || row_max == new_max) ? 1.f : exp2f(row_max - new_max);
        const float m_use = new_max == -INFINITY ? 0.f : new_max;
        row_max = new_max;
        // (the products up to tile j - 1 are through: the commit that S came with stands behind them)
        if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
          row_sum *= corr;
#pragma unroll
          for (int c = 0; c < DV / 32; ++c) {
            uint32_t ov[32];
            tmem_ld_32x32b_x32(o_col + c * 32, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
            tmem_st_32x32b_x32(o_col + c * 32, ov);
          }
        }
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (half == 1 && !whole) break;
          uint32_t pk[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const float a = exp2f(fmaf(__uint_as_float(sv[half * 2 + (c >> 4)][(2 * c) & 31]), scale, -m_use));
            const float b = exp2f(fmaf(__uint_as_float(sv[half * 2 + (c >> 4)][(2 * c + 1) & 31]), scale, -m_use));
            sum[(c & 1) * 2] += a;
            sum[(c & 1) * 2 + 1] += b;
            pk[c] = pack_bf16x2(a, b);
          }
          tmem_st_32x32b_x32(s_col + half * 32, pk);
        }
        row_sum += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);
      }
      if (!ok) break;
      ok = !*abort_flag && mbar_wait(&o_done[t], oc & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++oc;
      tc_fence_after_sync();
      const bool row_valid = m0 + r < it.q_len;
      const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
      __nv_bfloat16* dst = p.out + static_cast<long long>(it.q_begin + m0 + r) * p.out_stride +
                           static_cast<long long>(h) * DV;
#pragma unroll
      for (int c = 0; c < DV / 32; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32b_x32(o_col + c * 32, ov);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(ov[i * 8 + 0]) * inv, __uint_as_float(ov[i * 8 + 1]) * inv);
            v.y = pack_bf16x2(__uint_as_float(ov[i * 8 + 2]) * inv, __uint_as_float(ov[i * 8 + 3]) * inv);
            v.z = pack_bf16x2(__uint_as_float(ov[i * 8 + 4]) * inv, __uint_as_float(ov[i * 8 + 5]) * inv);
            v.w = pack_bf16x2(__uint_as_float(ov[i * 8 + 6]) * inv, __uint_as_float(ov[i * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + i * 8) = v;
          }
        }
      }
      if (p.lse && row_valid)
        p.lse[static_cast<long long>(it.q_begin + m0 + r) * p.Hq + h] =
            row_sum > 0.f ? (row_max + log2f(row_sum)) / kLog2e : -INFINITY;
      // O has been read: the arrival on p_full for the next item's first tile stands behind this
      tc_fence_before_sync();
    }
    if (!ok && lane == 0) give_up();
  }

  // ---- teardown: nothing may still be writing shared or tensor memory when the CTA leaves
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag && warp == 8 && lane == 0) {
    // copies still in flight land in this CTA's shared memory: wait (bounded) for the last one of each stage
    if (q_loads > 0) mbar_wait(q_full, (q_loads - 1) & 1);
    for (uint32_t c = k_loads > KS ? k_loads - KS : 0; c < k_loads; ++c) mbar_wait(&k_full[c % KS], (c / KS) & 1);
    for (uint32_t c = v_loads > VS ? v_loads - VS : 0; c < v_loads; ++c) mbar_wait(&v_full[c % VS], (c / VS) & 1);
  }
  if (warp == 9) {
    if (*abort_flag && lane == 0) {
      // products still in flight write tensor memory: wait (bounded) for them before it is freed
      tc_commit(drain_bar);
      mbar_wait(drain_bar, 0);
    }
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int DQK, bool FLAT>
static int launch_two_tiles(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p,
                            int box_rows, const TwoTileGrid& g, cudaStream_t stream) {
  auto kern = gqa_prefill_two_tiles_kernel<DQK, FLAT>;
  static_assert(two::Cfg<DQK>::SMEM <= 227 * 1024, "shared memory of an SM");
  static DeviceOnce once;
  int dev = 0;
  if (once.needed(&dev)) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return -22;
    if (fa.numRegs < two::MIN_REGS) return 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, two::Cfg<DQK>::SMEM) != cudaSuccess)
      return -20;
    once.mark(dev);
  }
  const int ctas = g.items < sm_count() ? g.items : sm_count();
  return launch_pdl(kern, dim3(ctas), dim3(two::THREADS), two::Cfg<DQK>::SMEM, stream, 1, tq, tk, tv, p, box_rows, g) ==
                 cudaSuccess
             ? 0
             : -21;
}

}  // namespace b200

using namespace b200;

// Returns 0 when the kernel ran, 1 when the problem is not one it takes (caller falls back), < 0 on error.
// Takes query / key head sizes 128 and 192 with value head size 128, no sliding window.
extern "C" int b200_gqa_prefill_tc(const void* q, const void* k_cache, const void* v_cache, void* out, float* lse,
                                   const int* block_tables, const int* cu_q, const int* seq_lens, int B,
                                   int max_q_len, int max_blocks, int block_size, int Hq, int Hk, int Dqk, int Dv,
                                   long long q_stride, long long out_stride, float scale, int causal, int window,
                                   long long total_q_rows, int num_cache_blocks, int* status, cudaStream_t stream) {
  if ((Dqk != 128 && Dqk != 192) || Dv != 128 || window != 0 || Hq % Hk != 0 || !(scale > 0.f)) return 1;
  const bool tma_ok = (block_size % 8) == 0 && (block_size <= 64 ? (64 % block_size) == 0 : (block_size % 64) == 0) &&
                      (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 && (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(q) & 15) == 0 && ((q_stride * 2) & 15) == 0 &&
                      ((out_stride * 2) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  if (!tma_ok || num_cache_blocks <= 0 || total_q_rows <= 0) return 1;
  if (B <= 0 || max_q_len <= 0) return 0;
  AttnParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_cache = static_cast<const __nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<const __nv_bfloat16*>(v_cache);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.block_tables = block_tables;
  p.cu_q = cu_q;
  p.seq_lens = seq_lens;
  p.max_blocks = max_blocks;
  p.block_size = block_size;
  p.Hq = Hq;
  p.Hk = Hk;
  p.q_stride = q_stride;
  p.out_stride = out_stride;
  p.scale_log2 = scale * kLog2e;
  p.causal = causal;
  p.status = status;
  p.num_cache_blocks = num_cache_blocks;
  // rows of a copy: what a cache block and a key tile have in common
  const int box_rows = block_size <= 64 ? block_size : (block_size % 128 ? 64 : 128);
  CUtensorMap tq, tk, tv;
  int r = make_tensormap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, static_cast<uint64_t>(total_q_rows),
                            static_cast<uint64_t>(Hq) * Dqk, static_cast<uint64_t>(q_stride), two::BM, 64,
                            CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  const uint64_t rows = static_cast<uint64_t>(num_cache_blocks) * Hk * block_size;
  r = make_tensormap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k_cache, rows, Dqk, Dqk, box_rows, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 2000;
  r = make_tensormap_2d(&tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, v_cache, rows, 128, 128, box_rows, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 3000;
  TwoTileGrid g;
  // (a single row tile per sequence and SMs to spare: one query tile per CTA, its keys read twice.  A prompt of 128 tokens,
  // 32 + 8 heads, 10.5 us with two heads per CTA, 8.5 in this form.)
  g.by_head = (Hq / Hk) % 2 == 0 && !(max_q_len <= two::BM && static_cast<long long>(Hq) * B <= sm_count());
  const int unit = g.by_head ? two::BM : 2 * two::BM;
  g.m_units = (max_q_len + unit - 1) / unit;
  g.head_units = g.by_head ? Hq / 2 : Hq;
  g.B = B;
  const long long items = static_cast<long long>(g.m_units) * g.head_units * B;
  if (items > 0x7fffffffll) return 1;
  g.items = static_cast<int>(items);
  return Dqk == 128 ? launch_two_tiles<128, false>(tq, tk, tv, p, box_rows, g, stream)
                    : launch_two_tiles<192, false>(tq, tk, tv, p, box_rows, g, stream);
}

// Non-absorbed latent attention over up-projected keys and values in place: q [T, H, 192] (pitch q_stride), kv [rows,
// H, 256] (pitch kv_stride; 128 of the key, 128 of the value), pe [rows, 64] (pitch pe_stride); sequence b has seq_lens[b]
// keys from row kv_start[b] on.  out [T, H, 128], causal.  Returns 1 (nothing done) for scales, pitches and alignments that
// the kernel does not take.
extern "C" int b200_mla_prefill(const void* q, const void* kv, const void* pe, void* out, const int* kv_start,
                                const int* cu_q, const int* seq_lens, int B, int max_q_len, int H, long long rows,
                                long long total_q_rows, long long q_stride, long long kv_stride, long long pe_stride,
                                long long out_stride, float scale, int* status, cudaStream_t stream) {
  if (B <= 0 || max_q_len <= 0 || total_q_rows <= 0 || rows <= 0) return 0;
  const uintptr_t bases = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kv) |
                          reinterpret_cast<uintptr_t>(pe) | reinterpret_cast<uintptr_t>(out);
  if (H <= 0 || !(scale > 0.f) || rows > 0x7fffffffll || (bases & 15) != 0 ||
      ((q_stride | kv_stride | pe_stride | out_stride) & 7) != 0)
    return 1;
  AttnParams p{};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.block_tables = kv_start;
  p.cu_q = cu_q;
  p.seq_lens = seq_lens;
  p.max_blocks = 1;
  p.Hq = p.Hk = H;
  p.out_stride = out_stride;
  p.scale_log2 = scale * kLog2e;
  p.causal = 1;
  p.status = status;
  CUtensorMap tq, tk, tp;
  int r = make_tensormap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, static_cast<uint64_t>(total_q_rows),
                            static_cast<uint64_t>(H) * 192, static_cast<uint64_t>(q_stride), two::BM, 64,
                            CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 1000;
  r = make_tensormap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, kv, static_cast<uint64_t>(rows),
                        static_cast<uint64_t>(H) * 256, static_cast<uint64_t>(kv_stride), two::BN, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 2000;
  r = make_tensormap_2d(&tp, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pe, static_cast<uint64_t>(rows), 64,
                        static_cast<uint64_t>(pe_stride), two::BN, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r) return r - 3000;
  TwoTileGrid g;
  g.by_head = 0;
  g.m_units = (max_q_len + 2 * two::BM - 1) / (2 * two::BM);
  g.head_units = H;
  g.B = B;
  const long long items = static_cast<long long>(g.m_units) * H * B;
  if (items > 0x7fffffffll) return 1;
  g.items = static_cast<int>(items);
  return launch_two_tiles<192, true>(tq, tk, tp, p, two::BN, g, stream);
}
