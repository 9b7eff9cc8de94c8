// CUDA-core GEMM for fp32 operands and small grids (gemm_simt.cu serves the rest): the networks and matrices whose few
// tiles leave an SM with little to hide latency behind.
#include "common.cuh"
#include "simt_tile.h"

namespace b2 {
namespace {

// One element of C: scale, beta, ReLU or ReLU mask.
__device__ __forceinline__ void finish(const GemmDesc& g, int gm, int gn, float acc) {
  float v = g.alpha * acc;
  float* c = static_cast<float*>(g.C) + (long long)gm * g.ldc + gn;
  if (g.beta != 0.f) v += g.beta * *c;
  if (g.epilogue == EPI_RELU) v = v > 0.f ? v : 0.f;
  if (g.epilogue == EPI_MASK) v = __ldg(static_cast<const float*>(g.aux) + (long long)gm * g.ldaux + gn) > 0.f ? v : 0.f;
  *c = v;
}

// 32 k of one operand (BMN rows or columns) on their way from global to shared memory by cp.async, in the layout
// they have in memory: K contiguous, rows of 128 bytes whose 16-byte chunk c lies at c ^ (row & 7); else k-rows of BMN
// floats. What lies outside the matrix arrives as zeros. `vec`: base and rows are whole 16-byte pieces.
constexpr int SLAB = 32;
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int BMN, int NT, bool KMAJOR>
__device__ __forceinline__ void copy_slab(uint32_t dst, const float* base, long long ld, int mn0, int k0, int MN, int K,
                                          bool vec, int t) {
  constexpr int CHUNKS = KMAJOR ? SLAB / 4 : BMN / 4;  // 16-byte chunks of a row in shared memory
#pragma unroll
  for (int i = 0; i < BMN * SLAB / 4 / NT; ++i) {
    const int q = t + i * NT, row = q / CHUNKS, chunk = q % CHUNKS;
    const int mn = mn0 + (KMAJOR ? row : chunk * 4), k = k0 + (KMAJOR ? chunk * 4 : row);
    const uint32_t at = dst + (KMAJOR ? row * (SLAB * 4) + ((chunk ^ (row & 7)) << 4) : row * (BMN * 4) + chunk * 16);
    const bool in = mn < MN && k < K;
    const int left = in ? min(4, KMAJOR ? K - k : MN - mn) : 0;
    const float* src = in ? base + (KMAJOR ? mn * ld + k : k * ld + mn) : base;
    if (vec) {
      copy16(at, src, left * 4);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) copy4(at + 4 * j, j < left ? src + j : base, j < left ? 4 : 0);
    }
  }
}

// Four k of T rows (or columns) of this thread: lane l of the L that share the dimension has rows l, l + L, ... of the
// warp's part where K is contiguous, groups of four neighbouring ones else; either way a warp's read is one
// conflict-free line.
template <int T, int L, bool KMAJOR>
__device__ __forceinline__ int own(int l, int i) { return KMAJOR ? l + L * i : l * 4 + (i & 3) + (i >> 2) * (4 * L); }
template <int BMN, int T, int L, bool KMAJOR>
__device__ __forceinline__ void fetch4(float (&f)[4][T], const uint8_t* slab, int mn, int l, int c) {
  if (KMAJOR) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
      const int row = mn + own<T, L, true>(l, i);
      const float4 v = *reinterpret_cast<const float4*>(slab + row * (SLAB * 4) + ((c ^ (row & 7)) << 4));
      f[0][i] = v.x; f[1][i] = v.y; f[2][i] = v.z; f[3][i] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < T; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(slab + (c * 4 + k) * (BMN * 4) + (mn + own<T, L, false>(l, i)) * 4);
        f[k][i] = v.x; f[k][i + 1] = v.y; f[k][i + 2] = v.z; f[k][i + 3] = v.w;
      }
  }
}

// Register-blocked tile GEMM for small grids and for rows that are not whole 16-byte pieces; every sum in k order, one FMA
// per term, as in gemm_simt_kernel. A warp owns WM x WN elements, its lanes a grid of WM/TM by WN/TN. Bound by latency
// where the grid is small: the copies of two slabs are in flight while one is multiplied, no thread holds a slab in
// registers (71 to 163 of them, against 222), and small tiles put many warps on an SM. us, forward / weight
// gradient / input gradient, gemm_simt_kernel -> here: 300 x 300 x 2000 105/118/113 -> 51/51/53; 200 x 123 x 701 33/39/34 ->
// 25/23/27.
template <int BM, int BN, int TM, int TN, int WM, int WN, bool AK, bool BK>
__global__ void __launch_bounds__((BM / WM) * (BN / WN) * 32) gemm_f32_kernel(GemmDesc g, int vec_a, int vec_b) {
  constexpr int NT = (BM / WM) * (BN / WN) * 32, LM = WM / TM, LN = WN / TN, STAGES = 3;
  constexpr int A_BYTES = BM * SLAB * 4, STAGE = (BM + BN) * SLAB * 4;
  static_assert(LM * LN == 32 && LM <= 8 && LN <= 8, "lanes of a warp; more than 8 rows would meet in a bank");
  extern __shared__ __align__(128) uint8_t smem[];
  const float* __restrict__ A = static_cast<const float*>(g.A);
  const float* __restrict__ B = static_cast<const float*>(g.B);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int lm = lane / LN, ln = lane % LN;
  const int wm = (warp / (BN / WN)) * WM, wn = (warp % (BN / WN)) * WN;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const long long lda = AK ? g.sAm : g.sAk, ldb = BK ? g.sBn : g.sBk;
  const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int slabs = (g.K + SLAB - 1) / SLAB;
  auto copy = [&](int s) {
    if (s < slabs) {
      const uint32_t dst = ring + (uint32_t)(s % STAGES) * STAGE;
      copy_slab<BM, NT, AK>(dst, A, lda, m0, s * SLAB, g.M, g.K, vec_a, t);
      copy_slab<BN, NT, BK>(dst + A_BYTES, B, ldb, n0, s * SLAB, g.N, g.K, vec_b, t);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  float fa[2][4][TM], fb[2][4][TN];
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) copy(s);
  for (int s = 0; s < slabs; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // slab s is there for all threads, and all have left the one that the next copy overwrites
    copy(s + STAGES - 1);
    const uint8_t* a = smem + (s % STAGES) * STAGE;
    const uint8_t* b = a + A_BYTES;
    fetch4<BM, TM, LM, AK>(fa[0], a, wm, lm, 0);
    fetch4<BN, TN, LN, BK>(fb[0], b, wn, ln, 0);
#pragma unroll
    for (int c = 0; c < SLAB / 4; ++c) {
      if (c + 1 < SLAB / 4) {
        fetch4<BM, TM, LM, AK>(fa[(c + 1) & 1], a, wm, lm, c + 1);
        fetch4<BN, TN, LN, BK>(fb[(c + 1) & 1], b, wn, ln, c + 1);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(fa[c & 1][k][i], fb[c & 1][k][j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + wm + own<TM, LM, AK>(lm, i);
    if (gm >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + wn + own<TN, LN, BK>(ln, j);
      if (gn < g.N) finish(g, gm, gn, acc[i][j]);
    }
  }
}

template <int BM, int BN, int TM, int TN, int WM, int WN, bool AK, bool BK>
cudaError_t launch_f32(const GemmDesc& g, int va, int vb, cudaStream_t stream) {
  constexpr int NT = (BM / WM) * (BN / WN) * 32, SMEM = 3 * (BM + BN) * SLAB * 4;
  static_assert(SMEM <= 48 * 1024, "dynamic shared memory without an attribute");
  gemm_f32_kernel<BM, BN, TM, TN, WM, WN, AK, BK>
      <<<dim3((g.N + BN - 1) / BN, (g.M + BM - 1) / BM), NT, SMEM, stream>>>(g, va, vb);
  return cudaGetLastError();
}
template <bool AK, bool BK>
cudaError_t launch_f32_tile(const GemmDesc& g, int tile, int va, int vb, cudaStream_t stream) {
  if (tile == 1) return launch_f32<64, 64, 8, 4, 32, 32, AK, BK>(g, va, vb, stream);
  if (tile == 2) return launch_f32<64, 32, 4, 4, 32, 16, AK, BK>(g, va, vb, stream);
  return launch_f32<32, 32, 4, 4, 16, 32, AK, BK>(g, va, vb, stream);
}

bool whole_pieces(const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; }
bool whole_a(const GemmDesc& g) { return whole_pieces(g.A, g.sAk == 1 ? g.sAm : g.sAk); }
bool whole_b(const GemmDesc& g) { return whole_pieces(g.B, g.sBk == 1 ? g.sBn : g.sBk); }

int tile_of(const GemmDesc& g) {
  if (g.in_type != T_F32 || g.out_type != T_F32 || (g.sAk != 1 && g.sAm != 1) || (g.sBk != 1 && g.sBn != 1)) return 0;
  return f32_tile(g.M, g.N, whole_a(g) && whole_b(g), 148);
}

}  // namespace

bool gemm_f32_serves(const GemmDesc& g) { return tile_of(g) > 0; }

cudaError_t gemm_f32_launch(const GemmDesc& g, cudaStream_t stream) {
  const int tile = tile_of(g), va = whole_a(g), vb = whole_b(g);
  if (g.sAk == 1 && g.sBk == 1) return launch_f32_tile<true, true>(g, tile, va, vb, stream);
  if (g.sAk == 1) return launch_f32_tile<true, false>(g, tile, va, vb, stream);
  if (g.sBk == 1) return launch_f32_tile<false, true>(g, tile, va, vb, stream);
  return launch_f32_tile<false, false>(g, tile, va, vb, stream);
}

}  // namespace b2
