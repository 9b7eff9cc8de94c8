// CUDA-core GEMMs: the small ones of the fp32 parity path of the training step (large ones: gemm_split.cu) and
// the fallback for shapes the tensor-core kernels do not take (the N = 1 tail layer of the reference topology,
// mlp_bench_common.h:26).
//
// Stand in for the reference's cblas_sgemm calls (mlp_omp.cc:474,566,657):
// C = alpha * op(A) * op(B) + beta * C with fp32 accumulation. Three kernels:
//   gemm_simt_kernel    any shape; every sum runs in k order, one FMA per term (small grids: gemm_f32.cu)
//   gemm_narrow_kernel  N <= 16 with K contiguous in both operands (the forward GEMM of a
//                       narrow output layer): lanes split K
//   gemm_short_kernel   M <= 16 with N contiguous in B (the weight gradient of that layer): warps split K
#include <algorithm>

#include "common.cuh"
#include "simt_tile.h"

namespace b2 {
namespace {

template <typename T>
__device__ __forceinline__ float ldf(const T* p);
template <>
__device__ __forceinline__ float ldf<float>(const float* p) { return __ldg(p); }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}

__device__ __forceinline__ float ldplain(const float* p) { return *p; }
__device__ __forceinline__ float ldplain(const __nv_bfloat16* p) { return __bfloat162float(*p); }

template <typename T>
__device__ __forceinline__ void stf(T* p, float v);
template <>
__device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <>
__device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// One element of C: scale, beta, ReLU or ReLU mask, conversion.
template <typename TI, typename TO>
__device__ __forceinline__ void finish(const GemmDesc& g, int gm, int gn, float acc) {
  float v = g.alpha * acc;
  TO* c = static_cast<TO*>(g.C) + (long long)gm * g.ldc + gn;
  if (g.beta != 0.f) v += g.beta * ldplain(c);
  if (g.epilogue == EPI_RELU) v = v > 0.f ? v : 0.f;
  if (g.epilogue == EPI_MASK) v = ldf(static_cast<const TI*>(g.aux) + (long long)gm * g.ldaux + gn) > 0.f ? v : 0.f;
  stf(c, v);
}

// Two independent fp32 FMAs in one instruction (each rounded like fmaf).
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long dup2(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

// The BMN x BK part of one operand that a thread block multiplies next, on its way from global
// memory (registers) to shared memory (k-major rows of BMN elements). `kmajor`: k is the contiguous
// dimension in memory. `vec` (fp32 only): base and leading dimension are multiples of 16 bytes.
template <typename TI, int BMN, int BK, int NT>
struct Loader {
  static constexpr int E = BMN * BK / NT;  // elements per thread
  float r[E];

  __device__ __forceinline__ void load(const TI* base, long long s_mn, long long s_k, bool kmajor, bool vec, int mn0,
                                       int k0, int MN, int K, int t) {
    if (sizeof(TI) == 4 && vec) {
#pragma unroll
      for (int i = 0; i < E / 4; ++i) {
        const int q = t + i * NT;
        int mm, kk;
        if (kmajor) { mm = q / (BK / 4); kk = (q % (BK / 4)) * 4; } else { mm = (q % (BMN / 4)) * 4; kk = q / (BMN / 4); }
        const int gm = mn0 + mm, gk = k0 + kk;
        const TI* p = base + gm * s_mn + gk * s_k;
        if (kmajor ? (gm < MN && gk + 4 <= K) : (gm + 4 <= MN && gk < K)) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(p));
          r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            r[4 * i + j] = (kmajor ? (gm < MN && gk + j < K) : (gm + j < MN && gk < K)) ? ldf(p + j) : 0.f;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int idx = t + i * NT;
        int mm, kk;
        if (kmajor) { kk = idx % BK; mm = idx / BK; } else { mm = idx % BMN; kk = idx / BMN; }
        const int gm = mn0 + mm, gk = k0 + kk;
        r[i] = (gm < MN && gk < K) ? ldf(base + gm * s_mn + gk * s_k) : 0.f;
      }
    }
  }
  __device__ __forceinline__ void store(float (*s)[BMN + 4], bool kmajor, bool vec, int t) const {
    if (sizeof(TI) == 4 && vec) {
#pragma unroll
      for (int i = 0; i < E / 4; ++i) {
        const int q = t + i * NT;
        if (kmajor) {
          const int mm = q / (BK / 4), kk = (q % (BK / 4)) * 4;
#pragma unroll
          for (int j = 0; j < 4; ++j) s[kk + j][mm] = r[4 * i + j];
        } else {
          const int mm = (q % (BMN / 4)) * 4, kk = q / (BMN / 4);
          *reinterpret_cast<float4*>(&s[kk][mm]) = make_float4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int idx = t + i * NT;
        if (kmajor) s[idx % BK][idx / BK] = r[i];
        else s[idx / BMN][idx % BMN] = r[i];
      }
    }
  }
};

// Register-blocked tile GEMM. A thread owns TM x TN elements as groups of four rows and four columns
// BM/(TM/4) and BN/(TN/4) apart, so that a warp's shared-memory reads are contiguous. Rows are kept
// in pairs for fma.rn.f32x2. The next k-slab travels from global memory to registers while the
// present one is multiplied, and two shared buffers leave one barrier per slab.
// Bound by FMA issue and, at one or two blocks per SM, by latency. 1024^3 forward / weight gradient /
// input gradient: 232/260/255 us with 128 x 128 tiles on 64 SMs and loads not overlapped, 74/66/74 us
// (29-33 TFLOP/s) as 64 x 64 tiles of this kernel.
template <typename TI, typename TO, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(GemmDesc g, int vec_a, int vec_b) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int GM = TM / 4, GN = TN / 4;  // groups of four
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Bs[2][BK][BN + 4];
  const TI* __restrict__ A = static_cast<const TI*>(g.A);
  const TI* __restrict__ B = static_cast<const TI*>(g.B);
  const int t = threadIdx.x;
  const int tx = t % (BN / TN), ty = t / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const bool a_kmajor = (g.sAk == 1), b_kmajor = (g.sBk == 1);

  unsigned long long acc[TM / 2][TN];  // rows 2i and 2i + 1 of the thread's tile
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  Loader<TI, BM, BK, NT> la;
  Loader<TI, BN, BK, NT> lb;
  la.load(A, g.sAm, g.sAk, a_kmajor, vec_a, m0, 0, g.M, g.K, t);
  lb.load(B, g.sBn, g.sBk, b_kmajor, vec_b, n0, 0, g.N, g.K, t);
  la.store(As[0], a_kmajor, vec_a, t);
  lb.store(Bs[0], b_kmajor, vec_b, t);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < g.K; k0 += BK) {
    const bool more = k0 + BK < g.K;
    if (more) {
      la.load(A, g.sAm, g.sAk, a_kmajor, vec_a, m0, k0 + BK, g.M, g.K, t);
      lb.load(B, g.sBn, g.sBk, b_kmajor, vec_b, n0, k0 + BK, g.N, g.K, t);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      unsigned long long a[TM / 2];
#pragma unroll
      for (int i = 0; i < GM; ++i) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&As[buf][kk][i * (BM / GM) + ty * 4]);
        a[2 * i] = v.x;
        a[2 * i + 1] = v.y;
      }
#pragma unroll
      for (int jg = 0; jg < GN; ++jg) {
        const float4 bv = *reinterpret_cast<const float4*>(&Bs[buf][kk][jg * (BN / GN) + tx * 4]);
        const unsigned long long b[4] = {dup2(bv.x), dup2(bv.y), dup2(bv.z), dup2(bv.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < TM / 2; ++i) fma2(acc[i][jg * 4 + j], a[i], b[j]);
      }
    }
    if (more) {
      la.store(As[buf ^ 1], a_kmajor, vec_a, t);
      lb.store(Bs[buf ^ 1], b_kmajor, vec_b, t);
      __syncthreads();
      buf ^= 1;
    }
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + (i / 4) * (BM / GM) + ty * 4 + (i & 3);
    if (gm >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + (j / 4) * (BN / GN) + tx * 4 + (j & 3);
      if (gn >= g.N) continue;
      const unsigned long long pair = acc[i / 2][j];
      finish<TI, TO>(g, gm, gn, __uint_as_float((i & 1) ? (unsigned int)(pair >> 32) : (unsigned int)pair));
    }
  }
}

// N <= 16, K contiguous in A and B. A warp computes R rows of C; its lanes stride over K and the
// partial sums meet in a shuffle reduction. As a 128 x 128 tile such a layer occupied M/128 SMs with
// a serial chain of K/16 slabs (1024 x 1 x 1024: 209 us).
template <typename TI, typename TO, int NMAX, int R>
__global__ void __launch_bounds__(128) gemm_narrow_kernel(GemmDesc g) {
  const TI* __restrict__ A = static_cast<const TI*>(g.A);
  const TI* __restrict__ B = static_cast<const TI*>(g.B);
  const int lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * R;
  if (row0 >= g.M) return;
  float acc[R][NMAX];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int n = 0; n < NMAX; ++n) acc[r][n] = 0.f;
#pragma unroll 4
  for (int k = lane; k < g.K; k += 32) {
    float a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = row0 + r < g.M ? ldf(A + (row0 + r) * g.sAm + k) : 0.f;
#pragma unroll
    for (int n = 0; n < NMAX; ++n) {
      if (n < g.N) {
        const float b = ldf(B + n * g.sBn + k);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][n] = fmaf(a[r], b, acc[r][n]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int n = 0; n < NMAX; ++n) {
      if (n < g.N) {
        float v = acc[r][n];
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, s);
        if (lane == n && row0 + r < g.M) finish<TI, TO>(g, row0 + r, n, v);
      }
    }
  }
}

// M <= 16, N contiguous in B. A block computes 32 columns of C; each of its 16 warps takes every
// sixteenth k, and the warps' partial sums meet in shared memory.
template <typename TI, typename TO, int MMAX>
__global__ void __launch_bounds__(512) gemm_short_kernel(GemmDesc g) {
  __shared__ float part[16][MMAX][32];
  const TI* __restrict__ A = static_cast<const TI*>(g.A);
  const TI* __restrict__ B = static_cast<const TI*>(g.B);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  float acc[MMAX];
#pragma unroll
  for (int m = 0; m < MMAX; ++m) acc[m] = 0.f;
#pragma unroll 4
  for (int k = warp; k < g.K; k += 16) {
    const float b = col < g.N ? ldf(B + k * g.sBk + col) : 0.f;
#pragma unroll
    for (int m = 0; m < MMAX; ++m)
      if (m < g.M) acc[m] = fmaf(ldf(A + m * g.sAm + k * g.sAk), b, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < MMAX; ++m) part[warp][m][lane] = acc[m];
  __syncthreads();
  for (int m = warp; m < g.M; m += 16) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 16; ++w) v += part[w][m][lane];
    if (col < g.N) finish<TI, TO>(g, m, col, v);
  }
}

// Tile of gemm_simt_kernel, an index into SIMT_TILES. Measured, us: 1024^3 as 64 x 64 74, as 64 x 32 105; 512 x 512 x 2048
// (64 tiles of 64 x 64 on 148 SMs) 94 and 72.
constexpr SimtTile SIMT_TILES[4] = {{128, 128, 1.0}, {64, 64, 0.85}, {64, 32, 0.555}, {32, 32, 0.40}};
int simt_tile(int M, int N, int sms) { return fastest_tile(SIMT_TILES, 4, M, N, sms); }

bool narrow_form(const GemmDesc& g) { return g.N <= 16 && g.K >= 64 && g.sAk == 1 && g.sBk == 1; }
bool short_form(const GemmDesc& g) { return g.M <= 16 && g.K >= 64 && g.sBn == 1; }

template <typename TI, typename TO>
cudaError_t launch(const GemmDesc& g, cudaStream_t stream) {
  if (narrow_form(g)) {
    if (g.N <= 2) gemm_narrow_kernel<TI, TO, 2, 1><<<(g.M + 3) / 4, 128, 0, stream>>>(g);
    else gemm_narrow_kernel<TI, TO, 16, 2><<<(g.M + 7) / 8, 128, 0, stream>>>(g);
    return cudaGetLastError();
  }
  if (short_form(g)) {
    if (g.M <= 2) gemm_short_kernel<TI, TO, 2><<<(g.N + 31) / 32, 512, 0, stream>>>(g);
    else gemm_short_kernel<TI, TO, 16><<<(g.N + 31) / 32, 512, 0, stream>>>(g);
    return cudaGetLastError();
  }
  if (!g.large_tiles && gemm_f32_serves(g)) return gemm_f32_launch(g, stream);
  auto vec = [](const void* p, long long ld) {
    return sizeof(TI) == 4 && reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0 ? 1 : 0;
  };
  const int va = vec(g.A, g.sAk == 1 ? g.sAm : g.sAk), vb = vec(g.B, g.sBk == 1 ? g.sBn : g.sBk);
  const int tile = simt_tile(g.M, g.N, 148);
  const SimtTile& c = SIMT_TILES[tile];
  const dim3 grid((g.N + c.bn - 1) / c.bn, (g.M + c.bm - 1) / c.bm);
  if (tile == 0) gemm_simt_kernel<TI, TO, 128, 128, 16, 8, 8><<<grid, 256, 0, stream>>>(g, va, vb);
  else if (tile == 1) gemm_simt_kernel<TI, TO, 64, 64, 32, 8, 4><<<grid, 128, 0, stream>>>(g, va, vb);
  else if (tile == 2) gemm_simt_kernel<TI, TO, 64, 32, 32, 4, 4><<<grid, 128, 0, stream>>>(g, va, vb);
  else gemm_simt_kernel<TI, TO, 32, 32, 32, 4, 4><<<grid, 64, 0, stream>>>(g, va, vb);
  return cudaGetLastError();
}

}  // namespace

bool gemm_simt_small(const GemmDesc& g) { return narrow_form(g) || short_form(g) || gemm_f32_serves(g); }

// us: 4.5 and the longer of 24 (28 where rows are not whole 16-byte pieces) per 1000 k and the flops at 33 (30) TFLOP/s; narrow
// and short forms 15 and 76 per 1000 k, roughly (their columns and rows count too).
double gemm_simt_us(const GemmDesc& g) {
  if (narrow_form(g)) return 4.5 + 0.015 * g.K;
  if (short_form(g)) return 4.5 + 0.076 * g.K;
  auto whole = [](const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; };
  const bool a = g.sAk != 1 || whole(g.A, g.sAm), b = whole(g.B, g.sBk == 1 ? g.sBn : g.sBk);
  return 4.5 + std::max((a && b ? 0.024 : 0.028) * g.K, (double)g.M * g.N * g.K / (a && b ? 16.5e6 : 15e6));
}

bool gemm_simt_short_sums(const GemmDesc& g) { return narrow_form(g) || short_form(g); }

cudaError_t gemm_simt_launch(const GemmDesc& g, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  if (g.in_type == T_F32 && g.out_type == T_F32) return launch<float, float>(g, stream);
  if (g.in_type == T_BF16 && g.out_type == T_BF16) return launch<__nv_bfloat16, __nv_bfloat16>(g, stream);
  if (g.in_type == T_BF16 && g.out_type == T_F32) return launch<__nv_bfloat16, float>(g, stream);
  return cudaErrorInvalidValue;
}

}  // namespace b2
