// How the kernels that take the weights as the M operand deal the tiles of a grouped product to the groups: the groups'
// offsets lie on the device, so every CTA adds up the tiles ahead of each group for itself.
#pragma once

namespace b200 {

// One warp: prefix[e] = tiles of the groups before e, first_row[e] = offsets[e], for e in 0 .. E.  tiles_of(rows): tiles of a
// group of that many rows.
template <typename TilesOf>
__device__ __forceinline__ void group_tiles(const int* offsets, int E, int* prefix, int* first_row, TilesOf tiles_of) {
  const int lane = threadIdx.x & 31, per = (E + 31) / 32;
  const int e0 = min(E, lane * per), e1 = min(E, e0 + per);
  int tiles = 0;
  for (int e = e0; e < e1; ++e) tiles += tiles_of(offsets[e + 1] - offsets[e]);
  int incl = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  int before = incl - tiles;
  for (int e = e0; e < e1; ++e) {
    const int a = offsets[e], b = offsets[e + 1];
    prefix[e] = before;
    first_row[e] = a;
    before += tiles_of(b - a);
    if (e + 1 == E) {
      prefix[E] = before;
      first_row[E] = b;
    }
  }
}

}  // namespace b200
