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

}  // namespace b2
