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

}  // namespace b2
