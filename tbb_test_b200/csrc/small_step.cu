// Whole training steps of small fp32 networks in one launch.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace b2 {
namespace {

constexpr int GROUPS = 4, GROUP = 128, THREADS = GROUPS * GROUP;  // a group of four warps works on a tile of its own
constexpr int TILE_M = 16, TILE_N = 32;  // a thread: four rows of a column
constexpr int CHUNK = 64, STAGES = 4;    // k per stage: a trip to L2 takes as long as two or three are multiplied
// rows of CHUNK k, four words apart in banks, or of TILE_M and TILE_N elements of one k
constexpr int PITCH = CHUNK + 4, A_FLOATS = TILE_M * PITCH, B_FLOATS = TILE_N * PITCH, STAGE = A_FLOATS + B_FLOATS;
static_assert(A_FLOATS >= CHUNK * TILE_M && B_FLOATS >= CHUNK * TILE_N, "either layout");
constexpr int SMEM_BYTES = GROUPS * STAGES * STAGE * 4;

enum Form : int { FWD = SMALL_FWD, DGRAD = SMALL_DGRAD, WGRAD = SMALL_WGRAD };
struct Gemm {
  int M, N, K;
  const float *A, *B;  // FWD: A m x k, B n x k; DGRAD: A m x k, B k x n; WGRAD: A k x m, B k x n; rows dense
  int form, layer;
  bool vec;    // rows of both are whole 16-byte pieces
  bool short_sums;  // see tile_sums
  __device__ __forceinline__ int tiles() const { return ((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N); }
};

// `rows` rows of `width` floats (a multiple of 4), the matrix's row 0 at `base`, to shared memory by cp.async, which goes
// past L1 in pieces of 16 bytes (`vec`: rows are whole ones). What lies outside arrives as zeros.
template <int WIDTH>
__device__ __forceinline__ void copy_rows(uint32_t dst, int pitch, const float* base, int ld, int row0, int rows, int row_end, int col0,
                                          int col_end, bool vec, int t) {
  for (int i = t; i < rows * (WIDTH / 4); i += GROUP) {
    const int r = i / (WIDTH / 4), c = i % (WIDTH / 4) * 4, row = row0 + r, left = row < row_end ? col_end - col0 - c : 0;
    const float* p = left > 0 ? base + (long long)row * ld + col0 + c : base;
    const uint32_t at = dst + (uint32_t)(r * pitch + c) * 4;
    if (vec) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(p), "r"(max(0, min(left, 4)) * 4) : "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at + 4 * j), "l"(j < left ? p + j : base), "r"(j < left ? 4 : 0) : "memory");
    }
  }
}

// Four sums of this thread. In k order, one FMA per term, like those of gemm_simt_kernel and gemm_f32_kernel. The GEMMs that
// a launch of their own would give to gemm_narrow_kernel or gemm_short_kernel, whose sums are 32 or 16 partial ones
// and a tree, are summed in blocks of eight terms instead (SHORT), and what an addition of a block loses is kept. That is fewer
// roundings than in those kernels: 4.5 per term in the mean, in squares of their size relative to a term, against at least 5 and
// a half for each of the k / 32 or k / 16 terms of a partial sum. Relative error against 64 bits in k order / in their kernel /
// here: 512 signed terms 3.8e-7 / 9.1e-8 / 6.4e-8, 2048 positive ones 6.1e-7 / 4.6e-8 / 2.6e-8. us per step in k order, so, and in
// separate launches: 512-10, batch 2000 59, 66, 115; 512-512-512, batch 8 45, 48, 147. (As pairs of floats in one instruction: 65, 52.)
template <int FORM, bool SHORT>
__device__ __forceinline__ void tile_sums(const Gemm& g, int m0, int n0, float* sh, int group, int t, float (&acc)[4]) {
  constexpr int STEP = SHORT ? 8 : 4;
  const int warp = t >> 5, lane = t & 31, chunks = (g.K + CHUNK - 1) / CHUNK;
  const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(sh));
  float rest[4] = {0.f, 0.f, 0.f, 0.f};  // SHORT: what acc has lost
  auto copy = [&](int c) {
    if (c < chunks) {
      const uint32_t a = at + (c % STAGES) * (STAGE * 4), b = a + A_FLOATS * 4;
      const int k0 = c * CHUNK, ks = min(CHUNK, (g.K - k0 + STEP - 1) / STEP * STEP);
      if (FORM == WGRAD) copy_rows<TILE_M>(a, TILE_M, g.A, g.M, k0, ks, g.K, m0, g.M, g.vec, t);
      else copy_rows<CHUNK>(a, PITCH, g.A, g.K, m0, TILE_M, g.M, k0, g.K, g.vec, t);
      if (FORM == FWD) copy_rows<CHUNK>(b, PITCH, g.B, g.K, n0, TILE_N, g.N, k0, g.K, g.vec, t);
      else copy_rows<TILE_N>(b, TILE_N, g.B, g.N, k0, ks, g.K, n0, g.N, g.vec, t);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(GROUP) : "memory"); };
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) copy(c);
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    sync();  // chunk c is there for all, and all have left the one that the next copy overwrites
    copy(c + STAGES - 1);
    const float* a = sh + (c % STAGES) * STAGE;
    const float* b = a + A_FLOATS;
    const int ks = min(CHUNK, g.K - c * CHUNK);
#pragma unroll 4
    for (int k0 = 0; k0 < ks; k0 += STEP) {  // behind the last k there are zeros
      float part[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) part[i] = SHORT ? 0.f : acc[i];
#pragma unroll
      for (int k = k0; k < k0 + STEP; k += 4) {
        float x[4][4], y[4];  // [row][k]
        if (FORM == WGRAD) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(a + (k + j) * TILE_M + warp * 4);
            x[0][j] = v.x; x[1][j] = v.y; x[2][j] = v.z; x[3][j] = v.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(a + (warp * 4 + i) * PITCH + k);
            x[i][0] = v.x; x[i][1] = v.y; x[i][2] = v.z; x[i][3] = v.w;
          }
        }
        if (FORM == FWD) {
          const float4 v = *reinterpret_cast<const float4*>(b + lane * PITCH + k);
          y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) y[j] = b[(k + j) * TILE_N + lane];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) part[i] = fmaf(x[i][j], y[j], part[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (SHORT) {  // the error of a sum of two, itself a float (Knuth)
          const float s = acc[i] + part[i], p = s - acc[i];
          rest[i] += (acc[i] - (s - p)) + (part[i] - p);
          acc[i] = s;
        } else {
          acc[i] = part[i];
        }
      }
    }
  }
  if (SHORT) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (fabsf(rest[i]) <= 3.402823466e38f) acc[i] += rest[i];  // else the sum is not finite
  }
  sync();  // before the next tile's copies
}

// All blocks (a cooperative launch) have come here: thread 0 of each counts itself in and waits, with a limit, until the
// counter has gone `blocks` further. False when a wait gave up, here or elsewhere, or `before` says that an earlier launch's
// did: the counter is then behind the host's, and nothing is to be waited for until the host has set both back.
__device__ __forceinline__ bool grid_barrier(unsigned int* counter, unsigned int until, unsigned int* status, unsigned int before) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    bool ok = before == 0;
    if (ok) {
      __threadfence();
      atomicAdd(counter, 1u);
    }
    unsigned long long t0 = 0;
    unsigned int spins = 0;
    while (ok && (int)(ld_acquire_u32(counter) - until) < 0) {
      if ((++spins & 0xFF) == 0) {
        const unsigned long long now = globaltimer();
        if (t0 == 0) t0 = now;
        if (now - t0 > WAIT_LIMIT_NS) atomicCAS(status, 0u, STATUS_GRID_BARRIER);
        ok = ld_acquire_u32(status) == 0;
      }
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// The step's GEMMs run in phases with a grid barrier between: forward layer by layer, the output gradient and the loss in the
// last one's epilogue, then for l = L-1 .. -1 the input gradient of layer l beside the weight gradient of layer l + 1,
// whose epilogue updates the weights that the phase before was the last to read. A phase is a list of 16 x 32 tiles.
// Bound by the latency of a phase where there is little to multiply: a trip to L2 for the operands, 4 ns per k, the
// stores, the barrier's fence, its atomic and the trip that notices it, 2.9 us together; else by shared memory reads (eight lines
// for the 16 FMAs of four k), half the FMA rate. Us per step in a launch of its own (5 less in
// launches of many), against a launch per GEMM on four streams: 128-256-128-64, batch 32 37 and 70; 6 x 48, batch 167 57 and 115;
// 3 x 512, batch 16 76 and 243; 9 x 162, batch 151 109 and 216; 8 x 416, batch 140 175 and 227.
// Tried: sums split over 16 warps, which meet in shared memory (the same in small batches, other bits); one
// cluster of 16 SMs and its barrier (3.7 us per phase, and nine times fewer SMs: 88-232-288-504-144-88, batch 26 315, 73 here).
__global__ void __launch_bounds__(THREADS) small_step_kernel(const __grid_constant__ SmallStep s, int steps, float lr, unsigned int count,
                                                             unsigned int* counter, unsigned int* status) {
  extern __shared__ __align__(16) float smem[];
  __shared__ double loss_part[THREADS / 32];
  const int t = threadIdx.x % GROUP, group = threadIdx.x / GROUP, warp = t >> 5, lane = t & 31, rank = blockIdx.x, blocks = gridDim.x;
  const int L = s.L;
  auto vec = [](int a, int b) { return a % 4 == 0 && b % 4 == 0; };
  auto fwd = [&](int l) {
    const SmallLayer& y = s.layer[l];
    return Gemm{s.batch, y.fo, y.fi, y.in, y.w, FWD, l, vec(y.fi, y.fi), y.short_sums[FWD]};
  };
  auto dgrad = [&](int l) {
    const SmallLayer& y = s.layer[l];
    return Gemm{s.batch, y.fi, y.fo, y.dz, y.w, DGRAD, l, vec(y.fo, y.fi), y.short_sums[DGRAD]};
  };
  auto wgrad = [&](int l) {
    const SmallLayer& y = s.layer[l];
    return Gemm{y.fo, y.fi, s.batch, y.dz, y.in, WGRAD, l, vec(y.fo, y.fi), y.short_sums[WGRAD]};
  };
  float loss = 0.f;  // of the elements this thread finishes in the last forward phase
  // what an element's epilogue reads: its target, the activation it is masked by, its weight
  auto fetch = [&](const Gemm& g, int m, int n) {
    const SmallLayer& y = s.layer[g.layer];
    const float* p = g.form == FWD ? (g.layer == L - 1 && s.baseline ? s.target : nullptr) : g.form == WGRAD ? y.w : s.baseline && g.layer > 0 ? y.in : nullptr;
    return p && m < g.M && n < g.N ? __ldcg(p + (long long)m * g.N + n) : 1.f;
  };
  auto finish = [&](const Gemm& g, int m, int n, float v, float x) {
    const SmallLayer& y = s.layer[g.layer];
    const long long at = (long long)m * g.N + n;
    if (g.form == FWD) {
      if (g.layer < L - 1) {
        y.out[at] = s.baseline ? fmaxf(v, 0.f) : v;
      } else {
        y.out[at] = v;
        const float d = s.baseline ? v - x : v;
        y.dz[at] = s.baseline ? d * s.inv_batch : d;
        loss += 0.5f * d * d;
      }
    } else if (g.form == DGRAD) {
      y.dx[at] = x > 0.f ? v : 0.f;
    } else {
      y.dw[at] = v;
      y.w[at] = fmaf(-lr, v, x);
    }
  };
  auto phase = [&](const Gemm& g0, const Gemm& g1, int n1) {  // n1: tiles of g1
    const int n0 = g0.tiles(), tiles = n0 + n1;
    for (int tile = group * blocks + rank; tile < tiles; tile += GROUPS * blocks) {
      const Gemm& g = tile < n0 ? g0 : g1;
      const int i = tile < n0 ? tile : tile - n0, nb = (g.N + TILE_N - 1) / TILE_N, mt = i / nb * TILE_M, nt = (i - i / nb * nb) * TILE_N;
      const int m = mt + warp * 4, n = nt + lane;
      float acc[4] = {0.f, 0.f, 0.f, 0.f}, x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = fetch(g, m + j, n);
      float* const sh = smem + group * STAGES * STAGE;
      auto sums = [&](auto is_short) {
        constexpr bool S = decltype(is_short)::value;
        if (g.form == FWD) tile_sums<FWD, S>(g, mt, nt, sh, group, t, acc);
        else if (g.form == DGRAD) tile_sums<DGRAD, S>(g, mt, nt, sh, group, t, acc);
        else tile_sums<WGRAD, S>(g, mt, nt, sh, group, t, acc);
      };
      if (g.short_sums) sums(std::true_type());
      else sums(std::false_type());
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (m + j < g.M && n < g.N) finish(g, m + j, n, acc[j], x[j]);
    }
  };
  const unsigned int before = threadIdx.x == 0 ? __ldcg(status) : 0;  // (no acquire: it would hold up the first copies)
  auto barrier = [&] { return grid_barrier(counter, count += blocks, status, before); };
  for (int step = 0; step < steps; ++step) {
    if (rank == 0 && threadIdx.x == 0) *s.loss = 0.0;  // the additions follow behind a barrier
    if (L == 1 && !barrier()) return;
    for (int l = 0; l < L; ++l) {
      const Gemm g = fwd(l);
      loss = 0.f;
      phase(g, g, 0);
      if (l == L - 1) {
        double sum = loss;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        if (lane == 0) loss_part[threadIdx.x / 32] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
          for (int w = 1; w < THREADS / 32; ++w) sum += loss_part[w];
          atomicAdd(s.loss, sum * s.loss_scale);
        }
      }
      if (!barrier()) return;
    }
    for (int l = L - 1; l >= -1; --l) {
      const bool d = l > 0 || (l == 0 && s.input_grad), w = l + 1 < L;
      if (d && w) {
        const Gemm g0 = dgrad(l), g1 = wgrad(l + 1);
        phase(g0, g1, g1.tiles());
      } else if (d || w) {
        const Gemm g = d ? dgrad(l) : wgrad(l + 1);
        phase(g, g, 0);
      }
      if (!(l < 0 && step + 1 == steps) && !barrier()) return;
    }
  }
}

}  // namespace

int small_step_barriers(const SmallStep& s, int steps) { return steps * (2 * s.L + 1 + (s.L == 1)) - 1; }

namespace {

int tiles(int m, int n) { return ((m + TILE_M - 1) / TILE_M) * ((n + TILE_N - 1) / TILE_N); }

// Time of a step, us: for each phase 1.6 and the longer of what its tiles take on all SMs, 0.59 and 0.0111 per k each, and what
// a group of warps takes for its share of either GEMM's, 0.59 and 0.0172 per k a tile; 1.29 times the terms of k where rows are
// not whole 16-byte pieces. Within 0.82 and 1.21 of the time measured for 400 networks of 1 to 16 layers, 1 to 8192 wide, batches
// of 1 to 2048 (4 x 4096, batch 1 904 us, 1 ms estimated; the weights alone, read and written, are 2 x 67 MB each).
double step_us(const SmallStep& s, int sms) {
  struct Load { double all, longest; };
  auto gemm = [&](int m, int n, int k, bool whole) {
    const double of_k = k * (whole ? 1.0 : 1.29), n_tiles = tiles(m, n);
    return Load{n_tiles * (0.59 + 0.0111 * of_k) / sms, std::ceil(n_tiles / (GROUPS * sms)) * (0.59 + 0.0172 * of_k)};
  };
  auto phase = [](Load a, Load b) { return 1.6 + std::max(a.all + b.all, std::max(a.longest, b.longest)); };
  auto whole = [](int a, int b) { return a % 4 == 0 && b % 4 == 0; };
  double us = 0;
  Load above{0, 0};  // the weight gradient of the layer above
  for (int l = s.L - 1; l >= 0; --l) {
    const SmallLayer& y = s.layer[l];
    us += phase(gemm(s.batch, y.fo, y.fi, whole(y.fi, y.fi)), Load{0, 0});
    us += phase(l > 0 || s.input_grad ? gemm(s.batch, y.fi, y.fo, whole(y.fo, y.fi)) : Load{0, 0}, above);
    above = gemm(y.fo, y.fi, s.batch, whole(y.fo, y.fi));
  }
  return us + phase(above, Load{0, 0});
}

}  // namespace

int small_step_blocks(const SmallStep& s, int sms) {
  int most = 1;
  for (int l = 0; l < s.L; ++l) {
    const SmallLayer& y = s.layer[l];
    const int above = l + 1 < s.L ? tiles(s.layer[l + 1].fo, s.layer[l + 1].fi) : 0;
    most = std::max({most, tiles(s.batch, y.fo), tiles(y.fo, y.fi), tiles(s.batch, y.fi) + above});
  }
  return std::min(most, sms);
}

// Networks whose average GEMM has at most 48 million multiplications, 40 where rows are not whole 16-byte pieces: beyond,
// the tensor cores of gemm_split.cu outweigh the launches (us per step here and there, whole rows: 4 x 256, batch 762 (50
// million) 127 and 152; 192-608-..., batch 699 (55) 348 and 380; 8 x 384, batch 436 (64) 307 and 258; others: 7 layers of 39 to 356,
// batch 2044 (40) 438 and 569; 5 of 157 to 948, batch 303 (49) 202 and 239; 8 of 32 to 724, batch 924 (49) 376 and 335). A weight
// gradient's sum walks the batch on one SM, and batches above 2048 have not been weighed.
// Below that, large layers among small ones, which a GEMM each serves better: where the estimate of a step is 1.15 times the one of
// separate launches (`launches_us`), as both are that exact (2048-2048-32-..., 14 layers, batch 128 355 and 305; 541-493-2742-10,
// batch 56 186 and 154; 64-5504, batch 82 107 and 89; left here: 64-1920-32-448-2912-1440, batch 37 275 and 228, the worst of 330).
// Batches of up to 16 are always faster here, whatever the widths: gemm_short_kernel walks K with 16 warps (4 x 4096, batch 2
// 906 and 1197; 4 x 2048, batch 8 362 and 1087).
bool small_step_serves(const SmallStep& s, int sms, double launches_us) {
  double macs = 0;
  bool whole = true;
  for (int l = 0; l < s.L; ++l) {
    macs += (double)s.batch * s.layer[l].fi * s.layer[l].fo;
    whole = whole && s.layer[l].fi % 4 == 0 && s.layer[l].fo % 4 == 0;
  }
  return s.batch <= 2048 && macs <= s.L * (whole ? 48e6 : 40e6) && (s.batch <= 16 || step_us(s, sms) <= 1.15 * launches_us);
}

// Steps that take about 2 ms (a launch may hold every SM).
int small_step_steps(const SmallStep& s, int sms) { return std::max(1, std::min(64, (int)(2000 / step_us(s, sms)))); }

cudaError_t small_step_launch(const SmallStep& s, int blocks, int steps, float lr, unsigned int count, unsigned int* counter,
                              unsigned int* status, cudaStream_t stream) {
  void* args[] = {const_cast<SmallStep*>(&s), &steps, &lr, &count, &counter, &status};
  static std::mutex attr_mutex;
  static unsigned long long attr_set = 0;  // one bit per device ordinal
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!(attr_set >> (dev & 63) & 1ull)) {
      cudaError_t e = cudaFuncSetAttribute(small_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
      if (e != cudaSuccess) return e;
      attr_set |= 1ull << (dev & 63);
    }
  }
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(small_step_kernel), dim3(blocks), dim3(THREADS), args, SMEM_BYTES, stream);
}

}  // namespace b2
