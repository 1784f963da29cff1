// How the weight-streaming kernels (gemm_stream.cu, gemm_fp8_stream.cu) share a tile's K among the CTAs of a cluster.
#pragma once

#include "../common/ptx.cuh"

namespace b200 {

// CTAs per tile of 128 weight rows: as many (a power of two up to the portable cluster size) as keep all CTAs resident at
// two per SM, and within the caller's limit (0: none), with at least four slabs of K each.  A cluster lies in one part of the
// chip, so that fewer CTAs of larger ones are resident (of 296: 284 in clusters of four, 264 in clusters of eight): 9216 x 4096
// bf16, one row, 72 tiles in four parts takes 21.5 us and in two parts 16.2, 9472 x 7168 e4m3 22.0 and 17.0; 64 tiles of
// 8192 x 2048 bf16 in four 9.6 and in two 10.5.
// Depends on the weights alone, so that the result of a row does not depend on the number of rows.
inline int stream_splits(int n_tiles, int k_slabs, int max_ctas, int sms) {
  const int most = max_ctas > 0 && max_ctas < 2 * sms ? max_ctas : 2 * sms;
  int best = 1;
  for (int s = 2; s <= 8; s *= 2) {
    const int per = (k_slabs + s - 1) / s;
    const int room = s == 2 ? most : most < 2 * sms * 9 / 10 ? most : 2 * sms * 9 / 10;
    if (static_cast<long long>(n_tiles) * s <= room && per >= 4 && (s - 1) * per < k_slabs) best = s;
  }
  return best;
}

// Four neighbouring values of the CTAs' parts, in rank order; at: their address in this CTA's shared memory.
__device__ __forceinline__ void split_sum(uint32_t at, int splits, float (&sum)[4]) {
  float v[8][4];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[s][i] = 0.f;
    if (s < splits)
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v[s][0]), "=f"(v[s][1]), "=f"(v[s][2]), "=f"(v[s][3])
                   : "r"(mapa_shared(at, s))
                   : "memory");
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sum[i] = v[0][i];
#pragma unroll
    for (int s = 1; s < 8; ++s) sum[i] += v[s][i];
  }
}

}  // namespace b200
