// Tile shape of the tensor-core GEMM (gemm_tcgen05.cu), chosen by a cost model on the host.
#pragma once

namespace b2 {

struct TileChoice {
  int sub_m;  // 128-row blocks per tile
  int bn;     // columns
  int pair;   // the tile belongs to a pair of SMs (cta_group::2)
};

// Cost of a shape = waves of the persistent grid over `sms` SMs times a tile's area per SM divided by the rate the shape
// sustains relative to 128 x 256 (measured at 1024 x 4096 x 4096 and 8192 x 4096 x 4096, bf16 and tf32). Filling every SM
// is not the goal: 1024 x 4096 x 4096 bf16 takes 31 us as 64 pair tiles, 35 us as 128 x 256, 41 us as 128 x 128 on all SMs.
// Pair tiles against 256 x 256 per SM, us forward / weight / input gradient: 8192 x 4096 x 4096 bf16 179/195/178 against
// 193/191/193, tf32 359/375/359 against 372/362/371; 1024 x 4096 x 4096 tf32 53/55/53 against 63/60/60 (128 x 256);
// 2048 x 8192 x 8192 bf16 191/182/190 against 190/189/190.
//
// `shared`: kernels of another library may sit on some of the SMs while this one runs (a step whose gradients are
// exchanged). A pair needs both SMs of a TPC, so each such SM can cost one, and a GEMM of one wave then takes two.
// That has not been measured since the pair kernel became the faster one (this needs several GPUs), so such steps keep
// the shapes and the rates their measurements were made with: 256 x 256 on one SM first, no pairs.
inline TileChoice choose_tile(int M, int N, int sms, bool x3, bool pair_ok, bool shared) {
  struct Cand { int sub_m, bn, pair; double rate, rate_shared; };
  const Cand cands[5] = {{2, 256, 1, 1.08, 0.0}, {2, 256, 0, 1.0, 1.0}, {1, 256, 0, 1.0, 0.93}, {1, 128, 0, 0.74, 0.70},
                         {1, 64, 0, 0.42, 0.45}};
  auto tiles = [&](int rows, int n) { return (long long)((M + rows - 1) / rows) * ((N + n - 1) / n); };
  double best = 1e300;
  int best_i = 4;
  for (int i = 0; i < 5; ++i) {
    const Cand& c = cands[i];
    if (c.pair && (!pair_ok || shared || sms < 2 || M <= 128)) continue;
    if (c.bn / 2 >= N && c.bn > 64) continue;          // tile wider than twice the matrix
    if (x3 && (c.sub_m == 2 || c.bn == 256)) continue;  // twice the shared memory per stage: 128 x 128 at most
    const long long T = tiles(c.sub_m * 128, c.bn);
    double waves, area = (double)(c.sub_m * 128) * c.bn;
    if (c.pair) {
      waves = (double)((T + sms / 2 - 1) / (sms / 2));
      area /= 2;
    } else if (c.sub_m == 2) {
      // the last partial wave is handed out as 128-row halves when that fits in one wave
      const long long full = T / sms, rem = T % sms;
      waves = (double)full + (rem == 0 ? 0.0 : (T > sms && rem * 2 <= sms ? 0.5 : 1.0));
    } else {
      waves = (double)((T + sms - 1) / sms);
    }
    const double cost = waves * area / (shared ? c.rate_shared : c.rate);
    if (cost < best * 0.999) { best = cost; best_i = i; }
  }
  return {cands[best_i].sub_m, cands[best_i].bn, cands[best_i].pair};
}

}  // namespace b2
