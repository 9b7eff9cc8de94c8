// Tile choice of the CUDA-core GEMMs (gemm_simt.cu, gemm_f32.cu).
#pragma once

namespace b2 {

struct SimtTile { int bm, bn; double rate; };

// A launch takes as long as its fullest SM: rounds of the grid over the SMs times the tile's area, divided by the rate the
// tile sustains (a smaller tile reads more shared memory per FMA). The first tile also serves where the others would need
// more row blocks than a grid has.
inline int fastest_tile(const SimtTile* tiles, int count, int M, int N, int sms) {
  int best = 0;
  double best_cost = 1e300;
  for (int i = 0; i < count; ++i) {
    const SimtTile& c = tiles[i];
    if (i > 0 && (M + c.bm - 1) / c.bm > 65535) continue;  // row blocks are gridDim.y
    const long long T = (long long)((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn);
    const double cost = (double)((T + sms - 1) / sms) * c.bm * c.bn / c.rate;
    if (cost < best_cost) { best_cost = cost; best = i; }
  }
  return best;
}

// Tile of gemm_f32_kernel, an index into F32_TILES, or 0, gemm_simt_kernel: grids that 32 x 32 tiles serve best, and any small
// grid with rows that are not whole 16-byte pieces. Measured, us: 1024^3 as 64 x 64 72, 64 x 32 78, 32 x 32 84; 512 x 512 x 2048 86,
// 60 and 55. Larger grids keep gemm_simt_kernel, which needs fewer instructions per FMA; so do the aligned ones in between,
// as 512 x 512 x 2048 (72 there): as weight gradients beside larger GEMMs they lost in 64 x 32 (6 x 512, batch 1024 458 -> 729 us
// per step), and on their own they have not been weighed.
constexpr SimtTile F32_TILES[4] = {{128, 128, 1.0}, {64, 64, 0.85}, {64, 32, 0.79}, {32, 32, 0.635}};
inline int f32_tile(int M, int N, bool whole_pieces, int sms) {
  const int tile = fastest_tile(F32_TILES, 4, M, N, sms);
  if (tile == 3) return tile;
  return !whole_pieces && (long long)((M + 63) / 64) * ((N + 63) / 64) <= sms ? tile : 0;
}

}  // namespace b2
