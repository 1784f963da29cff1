// Token sampling on the device:
//   * greedy arg-max (lowest index wins ties),
//   * temperature + top-k + top-p sampling by the exponential-race (Gumbel-max)
//     method: the kept set is found with counters over the logits
//     (counts for top-k, probability mass for top-p), then the winner is
//     argmax(logit / T + Gumbel noise) over the kept tokens, noise from a
//     counter-based Philox4x32-10 generator keyed per row.
// No sort, no host round trip; suitable for CUDA-graph capture.
//
// Replaces npu_top_k_top_p_sample and the exponential-noise side stream
// (omni_npu/sample/ops/topk_topp_sampler.py:41-88).

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/device_once.h"

namespace b200 {

static constexpr int kSampleThreads = 1024;

template <typename T>
__device__ __forceinline__ float load_logit(const T* row, int i);
template <>
__device__ __forceinline__ float load_logit<float>(const float* row, int i) {
  return row[i];
}
template <>
__device__ __forceinline__ float load_logit<__nv_bfloat16>(const __nv_bfloat16* row, int i) {
  return __bfloat162float(row[i]);
}

// Order-preserving map float -> uint32 (larger float = larger key).
__device__ __forceinline__ uint32_t float_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct MaxIdx {
  float v;
  int i;
};
__device__ __forceinline__ MaxIdx better(MaxIdx a, MaxIdx b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ MaxIdx block_argmax(MaxIdx m, MaxIdx* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxIdx other;
    other.v = __shfl_xor_sync(0xffffffffu, m.v, o);
    other.i = __shfl_xor_sync(0xffffffffu, m.i, o);
    m = better(m, other);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = m;
  __syncthreads();
  MaxIdx t = (l < (blockDim.x >> 5)) ? red[l] : MaxIdx{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxIdx other;
    other.v = __shfl_xor_sync(0xffffffffu, t.v, o);
    other.i = __shfl_xor_sync(0xffffffffu, t.i, o);
    t = better(t, other);
  }
  __syncthreads();
  return t;
}

// Philox4x32-10 (Salmon et al., SC'11): 128-bit counter, 64-bit key.
__device__ __forceinline__ uint4 philox4x32(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}

template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
argmax_kernel(const T* __restrict__ logits, int* __restrict__ out, int V, long long stride) {
  __shared__ MaxIdx red[32];
  const T* row = logits + static_cast<long long>(blockIdx.x) * stride;
  MaxIdx m{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float v = load_logit<T>(row, i);
    if (v > m.v) {
      m.v = v;
      m.i = i;
    }
  }
  m = block_argmax(m, red);
  if (threadIdx.x == 0) out[blockIdx.x] = m.i == 0x7fffffff ? 0 : m.i;
}

// ---------------------------------------------------------------------------------------------- sampling
// A thread-block cluster of CTAS = 8, 4 or 1 CTAs per row.  Each CTA keeps its part of the row in shared memory, so
// that a row of 128 k fp32 logits is read from device memory once and the later passes (threshold of top-k,
// threshold of top-p, draw) run from shared memory on eight SMs.  One CTA of 1024 threads per row, reading
// the row from memory in every pass, took 615 us for 128 rows x 128256 (its histogram over the leading key bits
// put most of the vocabulary into some thirty counters, and one thread walked the 2048 counters); this form is
// bound by the passes over shared memory.
// A row of temperature alone needs no threshold and is drawn from as it is read, without shared memory.
// Fewer CTAs for short rows, whose time is the exchanges': see launch_sample.
static constexpr int kMaxRowCtas = 8;
static constexpr int kRowThreads = 512;
static constexpr int kBins = 2048;
static constexpr int kMaxKeys = kBins / 2;
static constexpr int kMaxSlice = 50 * 1024;     // logits of a slice that fit shared memory
// Rows of at most this many logits take one CTA, four CTAs.
static constexpr int kOneCtaRow = 8 * 1024, kFourCtaRow = 48 * 1024;

struct RowShared {
  union {
    float mass[kBins];           // of this CTA's slice
    uint32_t count[kBins];
    struct {                     // CTA 0, after the counters have been read: the logits of the chosen bin
      uint32_t key[kMaxKeys];
      float weight[kMaxKeys];
    } list;
  };
  MaxIdx top;                    // of this CTA's slice
  MaxIdx red[32];
  float warp_sum[kRowThreads / 32];
  // one entry per CTA, which writes it into every CTA's copy: weight of its bins, its first bin at the target, weight before it
  float share[kMaxRowCtas];
  int first[kMaxRowCtas];
  float before[kMaxRowCtas];
  int own_first;
  float own_before;
  // CTA 0's, read by all
  int num_keys;
  uint32_t threshold;
};

__device__ __forceinline__ uint32_t remote_smem(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t remote_u32(const void* p, int rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote_smem(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ void remote_store(const void* p, int rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote_smem(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ float remote_f32(const void* p, int rank) { return __uint_as_float(remote_u32(p, rank)); }
template <int CTAS>
__device__ __forceinline__ void cluster_barrier() {
  if constexpr (CTAS == 1)
    __syncthreads();
  else
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Best of the slices' entries (every thread of every CTA gets it); ends with all CTAs past the exchange.
template <int CTAS>
__device__ __forceinline__ MaxIdx row_best(MaxIdx m, RowShared* sh) {
  m = block_argmax(m, sh->red);
  if constexpr (CTAS > 1) {
    if (threadIdx.x == 0) sh->top = m;
    cluster_barrier<CTAS>();
#pragma unroll
    for (int r = 0; r < CTAS; ++r)
      m = better(m, MaxIdx{remote_f32(&sh->top.v, r), static_cast<int>(remote_u32(&sh->top.i, r))});
    cluster_barrier<CTAS>();
  }
  return m;
}

// One pass of counters over the slices: ``bin_of(x)`` in [0, kBins) grows as logits fall, or is negative for
// logits that take no part.  Finds the first bin at which the weight of the bins up to it reaches the target
// (``target`` times the whole weight if SHARE); bin = -1 if rounding keeps the sum below the target.  Every CTA adds up its
// part of the bins over the row's CTAs.  (One CTA adding up all of them, 32 words of the other CTAs'
// shared memory per thread, held the seven others up: 112.6 us for the mixture of 128 rows x 128256, 97.2 in this form.)
struct PassResult {
  int bin;
  float above, target;
};

template <int CTAS, bool MASS, bool SHARE, typename Load, typename Bin>
__device__ PassResult count_pass(Load load, int n, int rank, Bin bin_of, float target, float scale_log2, float max_scaled,
                                 RowShared* sh) {
  for (int i = threadIdx.x; i < kBins; i += kRowThreads) sh->count[i] = 0u;    // also 0.f
  __syncthreads();
  // the last bin takes whatever lies far below the maximum, often most of the row: added up in registers
  float far = 0.f;
  for (int i = threadIdx.x; i < n; i += kRowThreads) {
    const float x = load(i);
    const int b = bin_of(x);
    if (b < 0) continue;
    const float w = MASS ? exp2f(__fmaf_rn(x, scale_log2, -max_scaled)) : 1.f;
    if (b == kBins - 1)
      far += w;
    else if (MASS)
      atomicAdd(&sh->mass[b], w);
    else
      atomicAdd(&sh->count[b], 1u);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) far += __shfl_xor_sync(0xffffffffu, far, o);
  if ((threadIdx.x & 31) == 0 && far > 0.f) {
    if (MASS)
      atomicAdd(&sh->mass[kBins - 1], far);
    else
      atomicAdd(&sh->count[kBins - 1], static_cast<uint32_t>(far));
  }
  cluster_barrier<CTAS>();
  constexpr int OWN = kBins / CTAS, PER = OWN > kRowThreads ? OWN / kRowThreads : 1;      // bins of a CTA, of a thread
  static_assert(OWN % PER == 0 && OWN / PER <= kRowThreads, "bins of the threads");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, bin0 = rank * OWN + threadIdx.x * PER;
  float w[PER], sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    w[i] = 0.f;
    if (threadIdx.x < OWN / PER) {
      uint32_t v[CTAS];
#pragma unroll
      for (int r = 0; r < CTAS; ++r) v[r] = CTAS == 1 ? sh->count[bin0 + i] : remote_u32(&sh->count[bin0 + i], r);
#pragma unroll
      for (int r = 0; r < CTAS; ++r) w[i] += MASS ? __uint_as_float(v[r]) : static_cast<float>(v[r]);
    }
    sum += w[i];
  }
  float incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) sh->warp_sum[warp] = incl;
  if (threadIdx.x == 0) {
    sh->own_first = 0x7fffffff;
    if (rank == 0) {
      sh->num_keys = 0;
      sh->threshold = 0u;
    }
  }
  __syncthreads();
  float run = incl - sum, own = 0.f;
#pragma unroll
  for (int i = 0; i < OWN / PER / 32; ++i) {
    if (i < warp) run += sh->warp_sum[i];
    own += sh->warp_sum[i];
  }
  if (threadIdx.x < CTAS) remote_store(&sh->share[rank], threadIdx.x, __float_as_uint(own));
  cluster_barrier<CTAS>();
  float total = 0.f;
#pragma unroll
  for (int r = 0; r < CTAS; ++r) {
    if (r < rank) run += sh->share[r];
    total += sh->share[r];
  }
  if (SHARE) target *= total;
  // an empty bin is never chosen; the smallest bin that qualifies is
  int mine = -1;
  float mine_before = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    if (mine < 0 && w[i] > 0.f && run + w[i] >= target) {
      mine = bin0 + i;
      mine_before = run;
    }
    run += w[i];
  }
  if (mine >= 0) atomicMin(&sh->own_first, mine);
  __syncthreads();
  if (mine >= 0 && sh->own_first == mine) sh->own_before = mine_before;
  __syncthreads();
  if (threadIdx.x < CTAS) {
    remote_store(&sh->first[rank], threadIdx.x, static_cast<uint32_t>(sh->own_first));
    remote_store(&sh->before[rank], threadIdx.x, __float_as_uint(sh->own_before));
  }
  cluster_barrier<CTAS>();
  PassResult res{-1, 0.f, target};
#pragma unroll
  for (int r = CTAS - 1; r >= 0; --r)
    if (sh->first[r] != 0x7fffffff) {
      res.bin = sh->first[r];
      res.above = sh->before[r];
    }
  return res;
}

// Largest key threshold such that the weight of the logits with key >= threshold is >= the target (as in
// count_pass), over the logits with key >= floor_key; 0 if there is none.  Weight: 1 or, MASS, exp2(x s - m).
// The first counters are linear in the logit (1/32 of a power of two of probability below the maximum), which
// spreads a vocabulary over them; the keys of the chosen bin are then compared with one another, or, if there are
// more than kMaxKeys of them (equal logits), go through counters of their key bits.
template <int CTAS, bool MASS, typename Load>
__device__ uint32_t row_threshold(Load load, int n, int rank, float target, uint32_t floor_key, float scale_log2,
                                  float max_scaled, RowShared* sh) {
  const auto linear = [=](float x) {
    const int b = static_cast<int>(__fmaf_rn(-x, scale_log2, max_scaled) * 32.f);
    return float_key(x) < floor_key ? -1 : min(max(b, 0), kBins - 1);
  };
  if (!(target > 0.f)) return 0xffffffffu;      // top_p <= 0: nothing qualifies, the caller falls back to the maximum
  const PassResult first = count_pass<CTAS, MASS, MASS>(load, n, rank, linear, target, scale_log2, max_scaled, sh);
  const int bin = first.bin;
  if (bin < 0) return 0u;
  target = first.target;
  float above = first.above;
  const uint32_t counter = remote_smem(&sh->num_keys, 0);
  for (int i = threadIdx.x; i < n; i += kRowThreads) {
    const float x = load(i);
    if (linear(x) != bin) continue;
    uint32_t at;
    asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(at) : "r"(counter) : "memory");
    if (at < kMaxKeys)
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote_smem(&sh->list.key[at], 0)), "r"(float_key(x))
                   : "memory");
  }
  cluster_barrier<CTAS>();
  const int found = static_cast<int>(remote_u32(&sh->num_keys, 0));
  if (found <= kMaxKeys) {
    if (rank == 0) {
      for (int i = threadIdx.x; i < found; i += kRowThreads) {
        const uint32_t key = sh->list.key[i];
        const float x = __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
        sh->list.weight[i] = MASS ? exp2f(__fmaf_rn(x, scale_log2, -max_scaled)) : 1.f;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < found; i += kRowThreads) {
        const uint32_t key = sh->list.key[i];
        float sum = above;
        uint32_t least = key;
#pragma unroll 4
        for (int j = 0; j < found; ++j) {
          const uint32_t other = sh->list.key[j];
          least = min(least, other);
          if (other >= key) sum += sh->list.weight[j];
        }
        // (the least key qualifies by the choice of the bin, whatever the order of the sums says)
        if (sum >= target || key == least) atomicMax(&sh->threshold, key);
      }
    }
    cluster_barrier<CTAS>();
    return remote_u32(&sh->threshold, 0);      // reset behind the first barrier of the next count_pass
  }
  uint32_t prefix = 0u, mask = 0u;
  for (int shift = 22; shift >= 0; shift = shift == 2 ? -1 : shift - 10) {
    // digits of 10, 10, 10 and the last 2 bits
    const auto digit = [=](float x) {
      const uint32_t key = float_key(x);
      return linear(x) != bin || (key & mask) != prefix ? -1 : 1023 - static_cast<int>((key >> shift) & 1023u);
    };
    const PassResult res = count_pass<CTAS, MASS, false>(load, n, rank, digit, target - above, scale_log2, max_scaled, sh);
    const int b = res.bin;
    if (b >= 0) above += res.above;
    const uint32_t d = b < 0 ? 0u : static_cast<uint32_t>(1023 - b);
    prefix |= d << shift;
    mask |= 1023u << shift;
  }
  const auto tail = [=](float x) {
    const uint32_t key = float_key(x);
    return linear(x) != bin || (key & mask) != prefix ? -1 : 3 - static_cast<int>(key & 3u);
  };
  const int b = count_pass<CTAS, MASS, false>(load, n, rank, tail, target - above, scale_log2, max_scaled, sh).bin;
  return prefix | (b < 0 ? 0u : static_cast<uint32_t>(3 - b));
}

struct DrawKey {
  uint2 key;
  uint32_t off_lo, off_hi;
};
__device__ __forceinline__ DrawKey draw_key(const long long* seeds, const long long* step_offset, int row) {
  const uint64_t seed = seeds ? static_cast<uint64_t>(seeds[row]) : 0x9E3779B97F4A7C15ull;
  const uint64_t off = step_offset ? static_cast<uint64_t>(step_offset[0]) : 0ull;
  return {make_uint2(static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32)), static_cast<uint32_t>(off),
          static_cast<uint32_t>(off >> 32)};
}

template <typename T, bool CACHED, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kRowThreads, 3)
sample_kernel(const T* __restrict__ logits, int* __restrict__ out, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const long long* __restrict__ seeds, const long long* __restrict__ step_offset, int V,
              long long stride, int slice) {
  extern __shared__ __align__(16) float cached[];
  __shared__ RowShared sh;
  const int rowi = blockIdx.x / CTAS;
  const int rank = blockIdx.x % CTAS;
  const int lo = min(V, rank * slice), n = min(V, lo + slice) - lo;
  const T* row = logits + static_cast<long long>(rowi) * stride + lo;
  const float temp = temperature ? temperature[rowi] : 1.f;
  const bool greedy = temp < 1e-5f;

  const int k = top_k ? top_k[rowi] : 0;
  const float p = top_p ? top_p[rowi] : 1.f;
  const bool by_count = k > 0 && k < V, by_mass = p < 1.f;

  // Gumbel-max over the kept set: four neighbours share a counter value
  MaxIdx best{-INFINITY, 0x7fffffff};
  const auto draw4 = [&](const DrawKey& d, const float (&x)[4], int i4, uint32_t floor_key) {
    const uint4 r = philox4x32(make_uint4(static_cast<uint32_t>(lo / 4 + i4), d.off_lo, d.off_hi, static_cast<uint32_t>(rowi)),
                               d.key);
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = lo + i4 * 4 + j;
      if (i4 * 4 + j >= n || float_key(x[j]) < floor_key) continue;
      // u in (0,1]; e = -log(u) ~ Exp(1); score = x/T - log(e)
      const float u = (static_cast<float>(rr[j] >> 8) + 1.0f) * (1.0f / 16777216.0f);
      const float e = -__logf(u);
      const float score = x[j] / temp - __logf(fmaxf(e, 1e-30f));
      if (score > best.v || (score == best.v && i < best.i)) {
        best.v = score;
        best.i = i;
      }
    }
  };

  // the maximum (the greedy answer), and the slice into shared memory
  MaxIdx m{-INFINITY, 0x7fffffff};
  const auto see = [&](float v, int i) {
    if (v > m.v) {
      m.v = v;
      m.i = i;
    }
  };
  int i0 = 0;
  const bool by_four = sizeof(T) == 4 && (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  if (!greedy && !by_count && !by_mass) {
    // every token stays: drawn from as it is read
    const DrawKey d = draw_key(seeds, step_offset, rowi);
#pragma unroll 2
    for (int i4 = threadIdx.x; i4 * 4 < n; i4 += kRowThreads) {
      float x[4];
      if (by_four && i4 * 4 + 3 < n) {
        const float4 v = reinterpret_cast<const float4*>(row)[i4];
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = i4 * 4 + j < n ? load_logit<T>(row, i4 * 4 + j) : -INFINITY;
      }
      draw4(d, x, i4, 0u);
    }
    best = row_best<CTAS>(best, &sh);
    if (rank == 0 && threadIdx.x == 0) out[rowi] = best.i == 0x7fffffff ? 0 : best.i;
    return;
  }
  if (by_four) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int n4 = n / 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < n4; i += kRowThreads) {
      const float4 v = row4[i];
      if (CACHED && !greedy) reinterpret_cast<float4*>(cached)[i] = v;
      see(v.x, lo + 4 * i);
      see(v.y, lo + 4 * i + 1);
      see(v.z, lo + 4 * i + 2);
      see(v.w, lo + 4 * i + 3);
    }
    i0 = n4 * 4;
  }
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < n; i += kRowThreads) {
    const float v = load_logit<T>(row, i);
    if (CACHED && !greedy) cached[i] = v;
    see(v, lo + i);
  }
  m = row_best<CTAS>(m, &sh);
  if (greedy) {
    if (rank == 0 && threadIdx.x == 0) out[rowi] = m.i == 0x7fffffff ? 0 : m.i;
    return;
  }
  const auto load = [&](int i) { return CACHED ? cached[i] : load_logit<T>(row, i); };
  const float scale_log2 = 1.4426950408889634f / temp;
  const float max_scaled = m.v * scale_log2;

  uint32_t floor_key = 0;  // keep keys >= floor_key
  if (by_count)
    floor_key = row_threshold<CTAS, false>(load, n, rank, static_cast<float>(k), 0u, scale_log2, max_scaled, &sh);
  if (by_mass)
    floor_key = max(floor_key, row_threshold<CTAS, true>(load, n, rank, p, floor_key, scale_log2, max_scaled, &sh));

  const DrawKey d = draw_key(seeds, step_offset, rowi);
  for (int i4 = threadIdx.x; i4 * 4 < n; i4 += kRowThreads) {
    float x[4];
    bool any = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[j] = i4 * 4 + j < n ? load(i4 * 4 + j) : 0.f;
      any |= i4 * 4 + j < n && float_key(x[j]) >= floor_key;
    }
    if (any) draw4(d, x, i4, floor_key);
  }
  best = row_best<CTAS>(best, &sh);
  if (rank == 0 && threadIdx.x == 0) out[rowi] = best.i == 0x7fffffff ? (m.i == 0x7fffffff ? 0 : m.i) : best.i;
}

template <typename T, bool CACHED, int CTAS>
int launch_sample_as(const void* logits, int* out, const float* temperature, const int* top_k, const float* top_p,
                     const long long* seeds, const long long* step_offset, int B, int V, long long stride, int slice,
                     cudaStream_t stream) {
  const auto kern = sample_kernel<T, CACHED, CTAS>;
  static DeviceOnce once;
  int dev = 0;
  if (CACHED && once.needed(&dev)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSlice * 4) != cudaSuccess) return -4;
    once.mark(dev);
  }
  kern<<<B * CTAS, kRowThreads, CACHED ? slice * 4 : 0, stream>>>(static_cast<const T*>(logits), out, temperature, top_k,
                                                                 top_p, seeds, step_offset, V, stride, slice);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <typename T>
int launch_sample(const void* logits, int* out, const float* temperature, const int* top_k, const float* top_p,
                  const long long* seeds, const long long* step_offset, int B, int V, long long stride,
                  cudaStream_t stream) {
  const int ctas = V <= kOneCtaRow ? 1 : V <= kFourCtaRow ? 4 : 8;
  // slices begin at a multiple of the four logits that share a draw
  const int slice = ((V + ctas - 1) / ctas + 3) / 4 * 4;
  const auto launch = ctas == 1            ? launch_sample_as<T, true, 1>
                      : ctas == 4          ? launch_sample_as<T, true, 4>
                      : slice <= kMaxSlice ? launch_sample_as<T, true, 8>
                                           : launch_sample_as<T, false, 8>;
  return launch(logits, out, temperature, top_k, top_p, seeds, step_offset, B, V, stride, slice, stream);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_argmax(const void* logits, int* out, int B, int V, long long stride,
                           int is_fp32, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (is_fp32)
    argmax_kernel<float><<<B, kSampleThreads, 0, stream>>>(static_cast<const float*>(logits), out, V, stride);
  else
    argmax_kernel<__nv_bfloat16><<<B, kSampleThreads, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(logits), out, V, stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

extern "C" int b200_sample(const void* logits, int* out, const float* temperature, const int* top_k,
                           const float* top_p, const long long* seeds, const long long* step_offset,
                           int B, int V, long long stride, int is_fp32, cudaStream_t stream) {
  if (B <= 0) return 0;
  return is_fp32 ? launch_sample<float>(logits, out, temperature, top_k, top_p, seeds, step_offset, B, V, stride, stream)
                 : launch_sample<__nv_bfloat16>(logits, out, temperature, top_k, top_p, seeds, step_offset, B, V,
                                                stride, stream);
}
