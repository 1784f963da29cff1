// Epilogue of the kernels that take the weights as the M operand: a lane holds one column of C (lane 0 a multiple of
// 32) and 16 consecutive rows of it.  Neighbouring lanes exchange values so that each stores two columns of every other
// row: half as many stores, of 4 bytes.  (One 2-byte store per row and lane, with the activation chosen inside the row
// loop, took 230 clocks a row, a single warp's chain of latencies: 14.4 us instead of 5.8 for a 64-row tile.)
#pragma once

#include "gated_act.cuh"

namespace b200 {

__device__ __forceinline__ uint32_t columns_pack(float lo, float hi) {
  __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&t);
}

// v: the lane's values of 16 rows, of which the first `rows` (the same for all lanes) exist; C: the first of these rows; n: the lane's column.
// Single columns (ACT: a unary activation, or none).
template <typename Act>
__device__ __forceinline__ void store_columns(const float (&v)[16], __nv_bfloat16* C, long long ldc, int n, int N, int rows,
                                              bool pairs, Act act) {
  if (pairs) {
    const int odd = n & 1;
    const bool ok = (n | 1) < N;
    __nv_bfloat16* dst = C + odd * ldc + (n & ~1);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      if (i >= rows) break;
      const float a = act(v[i]), b = act(v[i + 1]);
      const float other = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
      const uint32_t w = odd ? columns_pack(other, b) : columns_pack(a, other);
      if (ok && i + odd < rows) *reinterpret_cast<uint32_t*>(dst + i * ldc) = w;
    }
  } else if (n < N) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < rows) C[i * ldc + n] = __float2bfloat16(act(v[i]));
  }
}

// Gate and up columns alternate in groups of eight (N a multiple of 16); C has N / 2 columns.  A gate's lane computes
// row i, its up lane row i + 1.
template <typename Act>
__device__ __forceinline__ void store_gated_columns(const float (&v)[16], __nv_bfloat16* C, long long ldc, int n, int N,
                                                    int rows, bool pairs, Act act) {
  const int up = (n >> 3) & 1, odd = n & 1;
  const int col = (n >> 4) * 8 + (n & 7);
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    if (i >= rows) break;
    float o[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float a = v[i + 2 * j], b = v[i + 2 * j + 1];
      const float other = __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
      o[j] = up ? act(other, b) : act(a, other);
    }
    if (pairs) {
      // an even lane keeps rows i and i + 1, an odd lane rows i + 2 and i + 3
      const float other = __shfl_xor_sync(0xffffffffu, odd ? o[0] : o[1], 1);
      const uint32_t w = odd ? columns_pack(other, o[1]) : columns_pack(o[0], other);
      const int r = i + up + 2 * odd;
      if (n < N && r < rows) *reinterpret_cast<uint32_t*>(C + r * ldc + (col & ~1)) = w;
    } else if (n < N) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (i + 2 * j + up < rows) C[(i + 2 * j + up) * ldc + col] = __float2bfloat16(o[j]);
    }
  }
}

// fp32 results without an activation: the 32 lanes' values of a row are 128 neighbouring bytes as they are.
__device__ __forceinline__ void store_fp32_columns(const float (&v)[16], float* C, long long ldc, int n, int N, int rows) {
  if (n >= N) return;
  C += n;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (i < rows) C[i * ldc] = v[i];
}

// Whether two neighbouring columns can be stored as one word.
__device__ __forceinline__ bool columns_pair(const void* C, long long ldc, int N, bool gated) {
  return ((reinterpret_cast<uintptr_t>(C) & 3) == 0) && (ldc & 1) == 0 && (gated || (N & 1) == 0);
}

__device__ __forceinline__ void store_act_columns(int kind, float alpha, float limit, const float (&v)[16],
                                                  __nv_bfloat16* C, long long ldc, int n, int N, int rows, bool pairs) {
  if (kind == kActNone)
    store_columns(v, C, ldc, n, N, rows, pairs, [](float x) { return x; });
  else if (kind == kActSilu)
    store_gated_columns(v, C, ldc, n, N, rows, pairs, [](float g, float u) { return gated_act(kActSilu, g, u, 0.f, 0.f); });
  else if (act_is_gated(kind))
    store_gated_columns(v, C, ldc, n, N, rows, pairs,
                        [=](float g, float u) { return gated_act(kind, g, u, alpha, limit); });
  else
    store_columns(v, C, ldc, n, N, rows, pairs, [=](float x) { return unary_act(kind, x, alpha, limit); });
}

}  // namespace b200
