// Rules of the step kernel (step_kernel.cu, engine.cu): which networks run as whole steps, how many steps a launch takes,
// and which of its two forms serves.
#pragma once

namespace b2 {

enum StepPrec { STEP_BF16 = 0, STEP_TF32 = 1, STEP_X3 = 2 };

struct StepShape {
  const int* nf;    // widths, layers + 1 of them
  int layers, rows; // rows of the batch
  StepPrec prec;
  int sms;
  bool input_grad;  // the lowest layer's input gradient is computed
};

inline long long step_tiles(int m, int n, int bm, int bn) { return (long long)((m + bm - 1) / bm) * ((n + bn - 1) / bn); }

inline double step_flops(const StepShape& s) {
  double flops = 0;
  for (int l = 0; l < s.layers; ++l) flops += 6.0 * s.rows * s.nf[l] * s.nf[l + 1];
  return flops;
}
inline double step_flops_us(const StepShape& s) {  // all GEMMs at the rate the kernel reaches
  return step_flops(s) / (s.prec == STEP_BF16 ? 1000e6 : s.prec == STEP_X3 ? 200e6 : 500e6);
}

// Time of a step as one launch, us. The chain of layers: 4 us for each of its GEMMs, or what one CTA needs for a sum as long
// as the layer is wide. All GEMMs at the rate the kernel reaches, or all weights through the update, whichever is longer.
// And one weight gradient's sum over the batch, which one CTA walks alone. Estimated and measured: bf16 5 x 1024, batch 1024
// 76 and 89; 20 x 512, batch 2048 232 and 234; 4 x 64, batch 200000 771 and 838; 2 x 8192, batch 64 710 and 613; fp32-class
// 5 x 1024 257 and 227; 4 x 64, batch 200000 2930 and 3063. Over 160 networks the time measured
// is between 0.67 and 1.6 of it.
inline double step_us(const StepShape& s) {
  const int p = s.prec;
  const double chain_ns[3] = {2.8, 4.0, 8.0}, sum_ns[3] = {3.6, 6.5, 14.0};  // per term of a sum over a width, over the batch
  const double param_ps[3] = {4.6, 5.1, 7.6};                                // per weight, us per million
  double chain = 0, params = 0;
  for (int l = 0; l < s.layers; ++l) {
    for (int w : {s.nf[l], s.nf[l + 1]}) {
      const double sum = w * chain_ns[p] * 1e-3;
      chain += sum > 4.0 ? sum : 4.0;
    }
    params += (double)s.nf[l] * s.nf[l + 1];
  }
  const double work = step_flops_us(s), update = params * param_ps[p] * 1e-6;
  return chain + (work > update ? work : update) + s.rows * sum_ns[p] * 1e-3;
}

// Steps per launch, so that a launch lasts about LAUNCH_US, and a step at least: it holds every SM, and work of other
// handles, streams or processes gets its turn only between launches. Splitting costs nothing that shows: fp32-class 5 x 1024
// takes the same time per step in 22 launches as in 2 for 128 steps.
constexpr double LAUNCH_US = 2000.0;
inline int steps_per_launch(const StepShape& s) {
  const double n = LAUNCH_US / step_us(s);
  return n < 1 ? 1 : n > 64 ? 64 : (int)n;
}

// What the long sums of the chain leave idle: the terms of a sum times the share of SMs without a tile (128 x 64), over the
// forward and input-gradient GEMMs in the mean.
inline double step_idle_terms(const StepShape& s) {
  double idle = 0;
  int n = 0;
  auto gemm = [&](int cols, int sum) {
    const double share = 1.0 - (double)step_tiles(s.rows, cols, 128, 64) / s.sms;
    if (share > 0) idle += sum * share;
    ++n;
  };
  for (int l = 0; l < s.layers; ++l) {
    gemm(s.nf[l + 1], s.nf[l]);
    if (l > 0 || s.input_grad) gemm(s.nf[l], s.nf[l + 1]);
  }
  return n > 0 ? idle / n : 0;
}

// Whether steps run as one launch. Always where every GEMM is at most two rounds of 128 x 128 tiles over the SMs, however many
// layers there are (us per step, one launch per GEMM -> one for the step, fp32-class, 2048 wide, batch 2048: 16 layers 3853 ->
// 3154, 20 layers 4809 -> 3967). With larger GEMMs among them up to the size of an average GEMM from which on the larger
// tiles of gemm_tc_kernel (256 x 256 by CTA pairs; 128 x 128 in the fp32-class mode) outweigh the launch, fill and drain of
// every GEMM, and for steps of a few ms, since a launch holds every SM. By GFLOP of a GEMM: bf16 9 (800 wide, batch 8192) 292
// -> 173, 17 (1024, batch 8192) 436 -> 319, 25 (3072, batch 1300) 288 -> 263, 34 (2560, batch 2560) 316 -> 294, 34 (2048, batch
// 4096) 470 -> 473, 58 (3072, batch 3072) 426 -> 474; tf32 17 (4096, batch 512) 456 -> 381, 24 (2304, batch 2304) 439 -> 386
// but 25 (3072, batch 1300) 404 -> 439, 34 (2560, batch 2560) 501 -> 527; fp32-class 34 (2560) 1376 -> 1200, 69 (2048, batch
// 8192) 2753 -> 2427, 103 2793 -> 2423. One wide layer among narrow ones follows the average too: a 4096 x 4096 layer among
// ten of 64, batch 8192, bf16 1064 -> 892, among seven of 1024, batch 4096, 758 -> 701; an 8192 x 8192 layer among twenty of 256,
// batch 2048, 1218 -> 1179, tf32 1919 -> 1927; 4096 x 4096 among 24 of 512, batch 4096, tf32 2126 -> 1474. In bf16 the line is
// lower for layers that are not whole 128-byte columns, whose operands come in more boxes: 13 (900, batch 8000) 411 -> 337, 17
// (2040, batch 2040) 309 -> 302, but 23 (1700, batch 4000) 403 -> 431, 31 (2500, batch 2500) 386 -> 405, 30 (5000, batch 600) 550
// -> 591, and two layers of 9000 among four of 256, batch 1000, 823 -> 917; tf32 17 (2040) 421 -> 390, fp32-class 31 (2500) 1738
// -> 1581.
// Not where few tiles with long sums hold up the chain of layers (step_idle_terms): an SM that walks one takes its share of
// the weight gradients only afterwards, while separate launches let them fill the other SMs. By idle terms: bf16 6300 (1024-
// 16000-1024, batch 256) 273 -> 264, 7100 (batch 128) 252 -> 264, 9400 (2048-24000-2048, batch 128) 565 -> 606, 17800 (1024-
// 40000-1024, batch 128) 559 -> 653; tf32 5400 (1024-16000-1024, batch 300) 406 -> 388, 7100 371 -> 365, 9400 695 -> 770, 17800
// 895 -> 896; fp32-class 550 (4096, batch 256) 434 -> 397, 1100 (3072, batch 256) 298 -> 279, 2100 (batch 128) 265 -> 279, 2300
// (4096, batch 128) 375 -> 395, 3500 (1024-8000-1024, batch 128) 323 -> 342, 17800 1509 -> 1664.
inline bool step_serves(const StepShape& s) {
  bool short_gemms = true;
  for (int l = 0; l < s.layers; ++l) {
    const int in = s.nf[l], out = s.nf[l + 1];
    const long long most = 2LL * s.sms;
    if (step_tiles(s.rows, out, 128, 128) > most || step_tiles(out, in, 128, 128) > most ||
        ((l > 0 || s.input_grad) && step_tiles(s.rows, in, 128, 128) > most))
      short_gemms = false;
  }
  if (short_gemms) return true;
  double size = 0;  // of an average GEMM, 1 at the line
  for (int l = 0; l < s.layers; ++l) {
    const bool columns = s.nf[l] % 64 == 0 && s.nf[l + 1] % 64 == 0;
    const double most = s.prec == STEP_BF16 ? (columns ? 35e9 : 18e9) : s.prec == STEP_X3 ? 110e9 : 21e9;
    size += 2.0 * s.rows * s.nf[l] * s.nf[l + 1] / most / s.layers;
  }
  if (step_idle_terms(s) > (s.prec == STEP_X3 ? 2000 : 7000)) return false;
  return size <= 1.0 && 4.0 * 2 * s.layers + step_flops_us(s) <= 2 * LAUNCH_US;
}

// Whether the steps run on CTA pairs (256 x 128 tiles: a pair fetches 384 rows of operands where two 128 x 128 tiles fetch 512).
// Forward and input-gradient GEMMs of as many 128 x 128 tiles as fill the SMs, a little earlier where operands are 32 bits
// wide, gain by their flops; those of less than 48 tiles wait for latency, and smaller tiles on more SMs are shorter.
// us per step, one CTA per tile -> pairs, by tiles of a GEMM: 256 tiles (6 x 512, batch 8192) bf16 219 -> 171, tf32 411 -> 285;
// 256 (4 x 2048, batch 2048) bf16 222 -> 212, fp32-class 886 -> 804; 192 (6 x 1024, batch 3000) bf16 175 -> 156; 144 (4 x 1536,
// batch 1536) bf16 125 -> 129, tf32 195 -> 186; 128 (4 x 2048, batch 1024) bf16 156 -> 159, tf32 240 -> 222; 64 (5 x 1024, batch
// 1024) bf16 90 -> 95, fp32-class 233 -> 268. Mixed: 256 and 64 (2048-512-2048-512-2048, batch 2048) bf16 112 -> 105, tf32 173
// -> 151; 192 and 24 (2048-256-..., batch 1500) bf16 93 -> 104, tf32 141 -> 149, fp32-class 261 -> 277; 384 among 20 of 24
// (4096 x 4096 among layers of 256, batch 1500) bf16 288 -> 299, tf32 496 -> 484, fp32-class 1026 -> 988; 8192 x 8192 among
// layers of 64, batch 700, tf32 929 -> 840.
// Not where an odd number of row blocks, whose last pair is half empty, costs the chain a round over the SMs more: 12800 wide, batch
// 128, fp32-class 2402 -> 3052; 5000, batch 300, tf32 557 -> 617; 6144, batch 384, fp32-class 893 -> 1029 (bf16 loses without one
// at three blocks: 6400, batch 384 460 -> 486; five and more do not show: 4096, batch 640 331 -> 330).
inline bool step_pairs(const StepShape& s) {
  const int p = s.prec, blocks = (s.rows + 127) / 128;
  const double gain[3] = {0.075, 0.45, 0.6}, cost[3] = {1.0, 1.0, 1.5};  // us per GFLOP, us per GEMM
  if (s.sms < 2 || (p == STEP_BF16 && blocks == 3)) return false;
  const int fill = p == STEP_BF16 ? s.sms : s.sms * 2 / 3;
  double score = 0, single = 0, paired = 0;
  auto gemm = [&](int cols, int sum) {
    const long long tiles = step_tiles(s.rows, cols, 128, 128), pairs = step_tiles(s.rows, cols, 256, 128);
    if (tiles > fill) score += 2e-9 * s.rows * cols * sum * gain[p];
    else if (tiles < 48) score -= cost[p];
    single += (double)sum * ((tiles + s.sms - 1) / s.sms);
    paired += (double)sum * ((pairs + s.sms / 2 - 1) / (s.sms / 2));
  };
  for (int l = 0; l < s.layers; ++l) {
    gemm(s.nf[l + 1], s.nf[l]);
    if (l > 0 || s.input_grad) gemm(s.nf[l], s.nf[l + 1]);
  }
  return score > 0 && paired <= single;
}

}  // namespace b2
