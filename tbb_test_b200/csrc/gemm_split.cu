// GEMM on fp32 matrices whose products run on the tensor cores without giving up fp32 precision: every operand element
// is cut into three bf16 pieces that hold all of its 24 bits, and six of the nine products of pieces are summed.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace b2 {
namespace {

constexpr int BN = 64;       // columns of a tile; its rows are the 128 lanes of TMEM
constexpr int CHUNK_K = 64;  // elements of K per stage
constexpr int STAGES = 3;
// warps: sixteen load, cut and store the operands, eight add up the chunks and store C, one thread of the last issues the MMAs
constexpr int CUT_WARPS = 16, SUM_WARPS = 8, MMA_WARP = CUT_WARPS + SUM_WARPS, SPLIT_THREADS = (MMA_WARP + 1) * 32;
constexpr uint32_t B_PLANE = BN * 128;  // bytes of one piece of B's chunk
constexpr uint32_t B_STAGE = 3 * B_PLANE;
constexpr int SMEM_BYTES = 146 * 1024;  // the stages and what plain_part needs; one block per SM, whose whole TMEM it takes
// TMEM columns: D0, D1, D2, then the pieces of A's chunk (32 columns of two bf16 each) per stage
constexpr uint32_t T_D1 = BN, T_A = 3 * BN, A_HALF = 6 * 8, A_STAGE = 2 * A_HALF, T_ALL = 512;
static_assert(T_A + STAGES * A_STAGE <= T_ALL, "TMEM");

struct SplitParams {
  GemmDesc g;
  int how_ab, vec_c, vec_x;  // base and rows are whole pieces of 32 (2) or 16 (1) bytes
  int n_blocks, tiles;
  unsigned int* status;
};

__device__ __forceinline__ uint32_t to_bf16x2(float lo, float hi) {  // rounded to nearest even
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t to_six_bits(float lo, float hi) {  // to nearest: eight bits truncated and rounded once more
  uint32_t r;
  asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return (r + 0x00020002u) & 0xFFFCFFFCu;
}
// (lo, hi) - s * the bf16 pair p, exactly; s as two bf16.
__device__ __forceinline__ void take_off(float& lo, float& hi, uint32_t p, uint32_t minus_s) {
  asm("{\n\t.reg .b16 l, h, s, u;\n\tmov.b32 {l, h}, %2;\n\tmov.b32 {s, u}, %3;\n\t"
      "fma.rn.f32.bf16 %0, l, s, %0;\n\tfma.rn.f32.bf16 %1, h, s, %1;\n\t}"
      : "+f"(lo), "+f"(hi)
      : "r"(p), "r"(minus_s));
}
// Eight floats x as three bf16 pieces: x = h + 2^-16 (m + l), six bits in h and eight in m and l.
__device__ __forceinline__ void cut8(const float (&v)[8], uint32_t (&w)[3][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float x = v[2 * j], y = v[2 * j + 1];
    w[0][j] = to_six_bits(x, y);
    asm("{\n\t.reg .b64 a, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 s, {0f47800000, 0f47800000};\n\tmul.rn.f32x2 a, a, s;\n\t"
        "mov.b64 {%0, %1}, a;\n\t}"
        : "+f"(x), "+f"(y));
    take_off(x, y, w[0][j], 0xC780C780u);  // - 2^16 h
    w[1][j] = to_bf16x2(x, y);
    take_off(x, y, w[1][j], 0xBF80BF80u);  // - m
    w[2][j] = to_bf16x2(x, y);
  }
}

// How the next chunk is read: in groups of eight floats on 32-byte or 16-byte boundaries or float by float, all of them inside
// the matrix, or float by float with a check (CHECKED).
enum : int { CHECKED = -1, FLOATS = 0, BY16 = 1, BY32 = 2 };
// Eight neighbouring floats, of which `left` are inside the matrix; the rest is zero.
template <int HOW>
__device__ __forceinline__ void read8(const float* p, float (&r)[8], int left) {
  if (HOW == BY32) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "l"(p));
  } else if (HOW == BY16) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p)), v = __ldg(reinterpret_cast<const float4*>(p) + 1);
    r[0] = u.x; r[1] = u.y; r[2] = u.z; r[3] = u.w; r[4] = v.x; r[5] = v.y; r[6] = v.z; r[7] = v.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = HOW == FLOATS || j < left ? __ldg(p + j) : 0.f;
  }
}

// Where K is contiguous in A a lane reads eight k of a row and the lanes of a quad 32, whole 128-byte lines (as 16-byte
// reads of 64-byte pieces the loads took twice as many passes through L1, which bounded the kernel). The MMA's k-steps take
// four of the eight each, so the order of k in a k-step is 0-3, 8-11, 16-19, 24-27, and B is stored in the same order.
__device__ __forceinline__ int k_place(int k) { return (k & ~31) | (k & 4) << 2 | (k >> 1 & 12) | (k & 3); }

// A thread's 16 elements of the chunk of A, 128 rows by CHUNK_K, on their way from global memory through registers to
// three bf16 pieces in TMEM, lane = row, two k per column. Warp w has a part of rows 32 (w & 3) and k 32 (w >> 2 & 1) from on:
//   K contiguous: 16 rows; a lane eight k of two of them, eight rows apart (tcgen05.st 16x256b)
//   M contiguous: 16 k; a lane those of the row that is its number (32x32b)
// A stage is two halves of 32 k, each h, m, l of the first and the second k-step: 6 x 8 columns.
template <bool KMAJOR>
struct ShareA {
  const float* src;  // first element of the next chunk to load
  long long second;  // from part 0 to part 1
  int k;             // its position
  float r[2][8];

  __device__ __forceinline__ void begin(const GemmDesc& g, int m0, int t) {
    const int warp = t >> 5, lane = t & 31;
    // a row behind the last one stands for it: what comes of it is not stored
    const int row = m0 + (warp & 3) * 32 + (KMAJOR ? (warp >> 3) * 16 + (lane >> 2) : lane), m = min(row, g.M - 1);
    k = (warp >> 2 & 1) * 32 + (KMAJOR ? (lane & 3) * 8 : (warp >> 3) * 16);
    src = static_cast<const float*>(g.A) + m * g.sAm + k * g.sAk;
    second = KMAJOR ? (min(row + 8, g.M - 1) - m) * g.sAm : 8 * g.sAk;
  }
  __device__ __forceinline__ void advance(const GemmDesc& g) {
    src += g.sAk * CHUNK_K;
    k += CHUNK_K;
  }
  // part i: row + 8 i, or k + 8 i and on
  template <int HOW>
  __device__ __forceinline__ void load(const GemmDesc& g, int i) {
    const float* p = src + i * second;
    if (KMAJOR) {
      read8<HOW>(p, r[i], g.K - k);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j, p += g.sAk) r[i][j] = HOW != CHECKED || k + 8 * i + j < g.K ? __ldg(p) : 0.f;
    }
  }
  // first lane and column of warp w's part in a stage
  static __device__ __forceinline__ uint32_t offset(int w) {
    return ((uint32_t)((w & 3) * 32 + (KMAJOR ? (w >> 3) * 16 : 0)) << 16) + (uint32_t)((w >> 2 & 1) * A_HALF + (KMAJOR ? 0 : (w >> 3) * 8));
  }
  // Half i of the elements to TMEM: four k of either row, or eight k. The four words of a piece are one store, in the order the
  // cutting leaves them.
  __device__ __forceinline__ void store(uint32_t at, int i) const {
    uint32_t w[3][4];
    if (KMAJOR) {
      const float v[8] = {r[0][4 * i], r[0][4 * i + 1], r[0][4 * i + 2], r[0][4 * i + 3], r[1][4 * i], r[1][4 * i + 1], r[1][4 * i + 2], r[1][4 * i + 3]};
      cut8(v, w);
    } else {
      cut8(r[i], w);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      if (KMAJOR)
        asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16 * p + 8 * i), "r"(w[p][0]), "r"(w[p][1]),
                     "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
      else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16 * p + 4 * i), "r"(w[p][0]), "r"(w[p][1]),
                     "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
    }
  }
};

// A thread's eight neighbouring elements of the chunk of B, BN columns by CHUNK_K, on the same way to three pieces in
// shared memory: 128-byte rows (64 k of one column of C where K is contiguous, else 64 columns of one k), 128-byte swizzle.
template <bool KMAJOR, bool PLACED>
struct ShareB {
  const float* src;
  int n, k;
  bool inside;  // no group of eight lies outside in part
  float r[8];

  // (neighbouring groups of eight lanes store two rows apart, whose halves of a line do not meet in a bank)
  static __device__ __forceinline__ int row(int t) {
    return KMAJOR && PLACED ? (t >> 3 & ~3) | (t >> 3 & 1) << 1 | (t >> 4 & 1) : t >> 3;
  }
  __device__ __forceinline__ void begin(const GemmDesc& g, int n0, int t) {
    inside = KMAJOR || g.N % 8 == 0 || n0 + BN <= g.N;
    n = n0 + (KMAJOR ? row(t) : (t & 7) * 8);
    if (inside) n = min(n, g.N - (KMAJOR ? 1 : 8));
    k = KMAJOR ? (t & 7) * 8 : row(t);
    src = static_cast<const float*>(g.B) + n * g.sBn + k * g.sBk;
  }
  __device__ __forceinline__ void advance(const GemmDesc& g) {
    src += g.sBk * CHUNK_K;
    k += CHUNK_K;
  }
  template <int HOW>
  __device__ __forceinline__ void load(const GemmDesc& g) {
    read8<HOW>(src, r, KMAJOR ? g.K - k : k < g.K ? g.N - n : 0);
  }
  // offset of the group (its first half) in a piece
  static __device__ __forceinline__ uint32_t offset(int t) {
    const int at = KMAJOR ? row(t) : PLACED ? k_place(row(t)) : row(t);
    const int byte = KMAJOR && PLACED ? k_place((t & 7) * 8) * 2 : (t & 7) * 16;
    return at * 128 + ((byte & ~15) ^ (at & 7) << 4) + (byte & 15);
  }
  static __device__ __forceinline__ void store(uint32_t at, const uint32_t (&w)[3][4]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint32_t to = at + p * B_PLANE;
      if (KMAJOR && PLACED) {
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to), "r"(w[p][0]), "r"(w[p][1]) : "memory");
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to ^ 32), "r"(w[p][2]), "r"(w[p][3]) : "memory");
      } else {
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(w[p][0]), "r"(w[p][1]), "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
      }
    }
  }
};

// Sixteen accumulator columns of this lane's row; the registers hold them after tmem_wait.
__device__ __forceinline__ void tmem_ld(uint32_t addr, float (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
        "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait(float (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                 "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15])
               :
               : "memory");
}
// One MMA with A in TMEM.
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One element of C: scale, beta, ReLU or ReLU mask.
__device__ __forceinline__ void finish(const GemmDesc& g, int gm, int gn, float acc) {
  float v = g.alpha * acc;
  float* c = static_cast<float*>(g.C) + (long long)gm * g.ldc + gn;
  if (g.beta != 0.f) v += g.beta * *c;
  if (g.epilogue == EPI_RELU) v = v > 0.f ? v : 0.f;
  if (g.epilogue == EPI_MASK) v = __ldg(static_cast<const float*>(g.aux) + (long long)gm * g.ldaux + gn) > 0.f ? v : 0.f;
  *c = v;
}
// A warp's 32 rows of C from row m0 and 32 columns from n0 on, from shared memory of the warp's own, so that a store writes
// four whole 128-byte lines (a lane storing its own row, 32 bytes at a time, took 3100 clocks per tile).
constexpr int OUT_PITCH = 32 + 4;
__device__ __forceinline__ void finish_part(const SplitParams& p, int m0, int n0, const float* sh, int lane) {
  const GemmDesc& g = p.g;
  const int gn = n0 + (lane & 7) * 4;
#pragma unroll 4
  for (int i = 0; i < 32; i += 4) {
    const int row = i + (lane >> 3), gm = m0 + row, left = gm < g.M ? g.N - gn : 0;
    float4 w = *reinterpret_cast<const float4*>(sh + row * OUT_PITCH + (lane & 7) * 4);
    if (g.beta != 0.f || left < 4 || !p.vec_c || (g.epilogue == EPI_MASK && !p.vec_x)) {
      const float e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) finish(g, gm, gn + j, e[j]);
      continue;
    }
    w.x *= g.alpha; w.y *= g.alpha; w.z *= g.alpha; w.w *= g.alpha;
    if (g.epilogue == EPI_RELU) {
      w.x = fmaxf(w.x, 0.f); w.y = fmaxf(w.y, 0.f); w.z = fmaxf(w.z, 0.f); w.w = fmaxf(w.w, 0.f);
    } else if (g.epilogue == EPI_MASK) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(g.aux) + (long long)gm * g.ldaux + gn));
      w.x = a.x > 0.f ? w.x : 0.f; w.y = a.y > 0.f ? w.y : 0.f; w.z = a.z > 0.f ? w.z : 0.f; w.w = a.w > 0.f ? w.w : 0.f;
    }
    *reinterpret_cast<float4*>(static_cast<float*>(g.C) + (long long)gm * g.ldc + gn) = w;
  }
}

// The same part of C by FMAs in k order: 16 k of both operands at a time as k-rows of 32 by cp.async, the next ones under way
// while these are multiplied; a lane has eight rows and four columns. Bound by the twelve floats that a lane reads for 32 FMAs
// (more accumulators have no registers) and their latency. us, operands all NaN, forward / weight / input gradient, CUDA-core
// kernels, here, and here with a lane to a row and no loads ahead: 1024^3 73/65/69, 125/116/120, 204/508/333; 2048^3 434/425/427,
// 933/873/891, 1552/4026/2620. (All eight warps on one slab of 128 x 64: 113/112/110, but 1 to 3 % on finite operands.)
constexpr int PLAIN_K = 16, PLAIN_STAGE = 2 * PLAIN_K * OUT_PITCH, PLAIN_BYTES = 2 * PLAIN_STAGE * 4;
static_assert(PLAIN_BYTES >= 32 * OUT_PITCH * 4, "finish_part's room");
static_assert(SMEM_BYTES >= 1024 + STAGES * (int)B_STAGE + SUM_WARPS * PLAIN_BYTES, "shared memory");
template <bool KMAJOR>
__device__ __forceinline__ void plain_copy(uint32_t dst, const void* base, long long s_mn, long long s_k, int mn0, int mn_end, int k0, int k_end,
                                           int lane) {
  // K contiguous: a lane has one k of every other row, else every k of one
  int mn = mn0 + (KMAJOR ? lane >> 4 : lane), k = k0 + (KMAJOR ? lane & 15 : 0);
  const float* p = static_cast<const float*>(base) + mn * s_mn + k * s_k;
  uint32_t at = dst + (uint32_t)((k - k0) * OUT_PITCH + mn - mn0) * 4;
#pragma unroll 4
  for (int i = 0; i < 16; ++i) {
    const bool in = mn < mn_end && k < k_end;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at), "l"(in ? p : static_cast<const float*>(base)), "r"(in ? 4 : 0) : "memory");
    if (KMAJOR) {
      mn += 2;
      p += 2 * s_mn;
      at += 2 * 4;
    } else {
      ++k;
      p += s_k;
      at += OUT_PITCH * 4;
    }
  }
}
template <bool AK, bool BK>
__device__ __forceinline__ void plain_part(const GemmDesc& g, int m0, int n0, float* sh, int lane) {
  const uint32_t at = smem_u32(sh);
  auto copy = [&](int k0) {
    if (k0 < g.K) {
      const uint32_t to = at + (uint32_t)(k0 / PLAIN_K & 1) * (PLAIN_STAGE * 4);
      plain_copy<AK>(to, g.A, g.sAm, g.sAk, m0, g.M, k0, g.K, lane);
      plain_copy<BK>(to + PLAIN_K * OUT_PITCH * 4, g.B, g.sBn, g.sBk, n0, g.N, k0, g.K, lane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int row = (lane >> 3) * 8, col = (lane & 7) * 4;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  copy(0);
#pragma unroll 1
  for (int k0 = 0; k0 < g.K; k0 += PLAIN_K) {
    copy(k0 + PLAIN_K);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const float* const a = sh + (k0 / PLAIN_K & 1) * PLAIN_STAGE + row;
    const float* const b = sh + (k0 / PLAIN_K & 1) * PLAIN_STAGE + PLAIN_K * OUT_PITCH + col;
    const int end = min(PLAIN_K, g.K - k0);
#pragma unroll 2
    for (int k = 0; k < end; ++k) {
      const float4 u = *reinterpret_cast<const float4*>(a + k * OUT_PITCH), v = *reinterpret_cast<const float4*>(a + k * OUT_PITCH + 4);
      const float4 w = *reinterpret_cast<const float4*>(b + k * OUT_PITCH);
      const float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w}, y[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
    }
    __syncwarp();  // before the next copies
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<float4*>(sh + (row + i) * OUT_PITCH + col) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// x = h + 2^-16 (m + l) with bf16 h, m, l, each rounded to nearest: 6, 8 and 8 bits and a sign each, so nothing of x is lost, and the
// scale keeps the low pieces of a small x away from the denormal numbers. C = D0 + 2^-16 D1 + 2^-32 D2 with
//   D0 = sum h h'     D1 = sum h m' + m h' + h l' + l h'     D2 = sum m m' + m l' + l m'
// What is dropped (l l') is 2^-32 of a product. The tensor core truncates when it adds into an accumulator, so D0 holds one
// chunk of 64 k only: the sum warps add it to the sum they keep in registers, rounding to nearest. D1 and D2 run over all of K
// in TMEM, where a truncation is 2^-6 and 2^-12 of one in D0. And h has six bits, not the eight that a bf16 holds: products of
// twelve mostly fit whole into D0 beside larger ones, so that little is truncated. Truncation has one sign, and with eight bits in h sums
// came out 3.8e-8 (operands signed) to 6.6e-8 (positive) of themselves small in the mean, now 5.7e-9 to 1.7e-8; a number made of
// many results shows it (the loss of nine 538-wide layers without ReLU was off by 7.7e-7, now by 8e-8, with FMAs by 8e-8 to 1.5e-7).
// It takes three instructions for every pair instead of one, m l' and l m' among the products, and 3 % of a step of 5 x 1024. Error
// against 64 bits in the norm of the result, here / FMAs in k order, signed and positive: K = 64 4.0e-8 / 1.5e-7 and
// 5.0e-8 / 1.2e-7, K = 4096 2.0e-7 / 1.2e-6 and 1.2e-7 / 8.5e-7. But products are added 16 at a time against the largest
// of them: where large terms cancel early in k order, FMAs keep a small one that is rounded away here.
// 32 x 32 elements with one that is not finite in the end (an Inf or a NaN among the operands, whose pieces are NaN, or numbers
// from 2^112 on) are computed again by FMAs in k order, so they are what the CUDA-core kernels give.
//
// Per 16 k one thread issues h h', h m', h l' and m l' (BN columns each), m [h'|m'] and l [h'|m'] (into D1 and D2 side by side). A comes
// from TMEM, so that an MMA reads 2 KB of shared memory instead of 6 (with A in shared memory an MMA of 64 columns took 74
// clocks, 42 so). Tiles of 64 columns: D0, D1, D2 and three stages of A fill TMEM, and 1024 x 1024 fills 128 SMs.
// Bound by the instructions that cut the operands (10 per pair of floats) and the latency of a chunk from load to hand-over:
// 0.9 us per chunk, of which the MMAs are 0.65. So sixteen warps cut, each a small part: with eight of twice the share a chunk took
// 1.0 us, with the summing in the same warps 1.05, with the pieces of A in shared memory 1.1 (1.5 for 128 columns). Beside its chunks a
// tile takes 5.5 us of launch, first loads and epilogue (8 with checked first loads, the first chunk handed over behind the second
// one's cut, and lanes storing their own rows).
// us, forward / weight / input gradient, against gemm_simt_kernel, operands in L2: 1024^3 24/24/22 against 74/65/69, 2048^3
// 130/135/120 (143 TFLOP/s) against 435/426/428, 512^3 15/16/15 against 22/22/22. 5 x 1024, batch 1024: 298 us per step, 938 before.
template <bool AK, bool BK>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) gemm_split_kernel(const __grid_constant__ SplitParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], sum_full, sum_empty, tile_full, tile_empty;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const uint32_t smem = (smem_u32(smem_raw) + 1023) & ~1023u;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  volatile int* abort_flag = &abort_s;
  const GemmDesc& g = p.g;
  ShareA<AK> sa;
  ShareB<BK, AK> sb;
  auto begin = [&](int tile) {
    sa.begin(g, tile / p.n_blocks * 128, t);
    sb.begin(g, tile % p.n_blocks * BN, t);
  };
  auto how = [&](int c) { return sb.inside && (c + 1) * CHUNK_K <= g.K ? p.how_ab : CHECKED; };
  if (warp < CUT_WARPS) {  // on its way while the block sets up
    begin(blockIdx.x);
    auto load = [&](auto h) {
      sa.template load<decltype(h)::value>(g, 0);
      sa.template load<decltype(h)::value>(g, 1);
      sb.template load<decltype(h)::value>(g);
    };
    if (how(0) == BY32) load(std::integral_constant<int, BY32>());
    else load(std::integral_constant<int, CHECKED>());
  }
  if (t == MMA_WARP * 32) {
    abort_s = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], CUT_WARPS);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&sum_full, 1);
    mbar_init(&sum_empty, SUM_WARPS);
    mbar_init(&tile_full, 1);
    mbar_init(&tile_empty, SUM_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(T_ALL)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  const int chunks = (g.K + CHUNK_K - 1) / CHUNK_K;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);

  if (warp == MMA_WARP) {
    if (elect_one()) {
      // B: K contiguous: 8-row groups 1024 bytes apart, 32 bytes of K per MMA; else groups of 8 k, and columns of 64 one piece apart
      const uint64_t b0 = make_smem_desc(smem, BK ? 16 : B_PLANE, 1024, 2);
      constexpr uint32_t B_STEP = (BK ? 32 : 16 * 128) >> 4, BP = B_PLANE >> 4, KS = CHUNK_K / 16;
      constexpr uint32_t one = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)!BK << 16) | ((uint32_t)(BN >> 3) << 17) |
                               ((uint32_t)(128 >> 4) << 24);
      constexpr uint32_t two = one + ((uint32_t)(BN >> 3) << 17);
      const uint32_t d1 = tmem + T_D1;
      int s = 0;
      uint32_t phase = 0, n = 0, tile_phase = 1;  // n: chunks so far
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        for (int c = 0; c < chunks; ++c, ++n) {
          if (!mbar_wait(&full_bar[s], phase, abort_flag, p.status, 1u) ||
              !mbar_wait(&sum_empty, (n & 1) ^ 1, abort_flag, p.status, 2u)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a = tmem + T_A + (uint32_t)s * A_STAGE;
          const uint64_t b = b0 + (uint32_t)s * (B_STAGE >> 4);
          auto piece = [&](uint32_t ks, uint32_t i) { return a + (ks >> 1) * A_HALF + i * 16 + (ks & 1) * 8; };
#pragma unroll
          for (uint32_t ks = 0; ks < KS; ++ks) mma_ts(tmem, piece(ks, 0), b + ks * B_STEP, one, ks > 0);
          tc_commit(smem_u32(&sum_full));
          if (c == 0) {  // D1 and D2 of the tile before have been read
            if (!mbar_wait(&tile_empty, tile_phase, abort_flag, p.status, 3u)) { ok = false; break; }
            tc_fence_after();
            tile_phase ^= 1;
          }
#pragma unroll
          for (uint32_t ks = 0; ks < KS; ++ks) {
            mma_ts(d1, piece(ks, 1), b + ks * B_STEP, two, c > 0 || ks > 0);
            mma_ts(d1, piece(ks, 0), b + BP + ks * B_STEP, one, 1u);
            mma_ts(d1, piece(ks, 0), b + 2 * BP + ks * B_STEP, one, 1u);
            mma_ts(d1, piece(ks, 2), b + ks * B_STEP, two, 1u);
            mma_ts(d1 + BN, piece(ks, 1), b + 2 * BP + ks * B_STEP, one, 1u);
          }
          tc_commit(smem_u32(&empty_bar[s]));
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        tc_commit(smem_u32(&tile_full));
      }
    }
  } else if (warp >= CUT_WARPS) {
    constexpr int COLS = BN * 4 / SUM_WARPS;
    const int col = (warp - CUT_WARPS) / 4 * COLS;
    float acc[COLS], d[16];
    uint32_t n = 0, tile_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
#pragma unroll
      for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
      for (int c = 0; c < chunks; ++c, ++n) {
        if (!mbar_wait(&sum_full, n & 1, abort_flag, p.status, 4u)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < COLS; h += 16) {
          tmem_ld(lanes + col + h, d);
          tmem_wait(d);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[h + j] += d[j];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sum_empty);
      }
      if (!ok || !mbar_wait(&tile_full, tile_phase, abort_flag, p.status, 5u)) break;
      tile_phase ^= 1;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2 * COLS; h += 16) {  // 2^-16 D1, 2^-32 D2
        tmem_ld(lanes + T_D1 + (h < COLS ? 0 : BN) + col + h % COLS, d);
        tmem_wait(d);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[h % COLS + j] += d[j] * (h < COLS ? 0x1p-16f : 0x1p-32f);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tile_empty);
      const int m0 = tile / p.n_blocks * 128 + (warp & 3) * 32, n0 = tile % p.n_blocks * BN + col;
      bool bad = false;  // not finite
#pragma unroll
      for (int j = 0; j < COLS; ++j) bad = bad || !(fabsf(acc[j]) <= 3.402823466e38f);
      float* const sh = reinterpret_cast<float*>(smem_raw + SMEM_BYTES - (warp - CUT_WARPS + 1) * PLAIN_BYTES);
      __syncwarp();  // all lanes have read the part before
      if (__any_sync(0xFFFFFFFFu, bad)) {
        plain_part<AK, BK>(g, m0, n0, sh, lane);
      } else {
#pragma unroll
        for (int j = 0; j < COLS; j += 4)
          *reinterpret_cast<float4*>(sh + lane * OUT_PITCH + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
      }
      __syncwarp();
      finish_part(p, m0, n0, sh, lane);
    }
  } else {
    const uint32_t a_at = tmem + T_A + ShareA<AK>::offset(warp), b_at = smem + ShareB<BK, AK>::offset(t);
    // What has been stored of a chunk is there for the MMAs. Done before the next chunk is cut, behind the wait for its stage:
    // the loads of it, which are on their way, hide the wait for the stores.
    auto hand_over = [&](int s) {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
    };
    // The present chunk into stage s, and behind each part of it the same part of the next one from memory.
    auto store_and_load = [&](int s, int s_before, auto how) {
      constexpr int V = decltype(how)::value;
      if (s_before >= 0) hand_over(s_before);
      sa.store(a_at + (uint32_t)s * A_STAGE, 0);
      if (!AK) sa.template load<V>(g, 0);
      sa.store(a_at + (uint32_t)s * A_STAGE, 1);
      if (AK) sa.template load<V>(g, 0);
      sa.template load<V>(g, 1);
      uint32_t w[3][4];
      cut8(sb.r, w);
      sb.store(b_at + (uint32_t)s * B_STAGE, w);
      sb.template load<V>(g);
    };
    int s = 0, s_before = -1;  // stage, and the one that is still to be handed over
    bool before_first = true;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
      for (int c = 0; c < chunks; ++c) {
        int next = c + 1;
        if (next < chunks) {
          sa.advance(g);
          sb.advance(g);
        } else if (tile + (int)gridDim.x < p.tiles) {
          begin(tile + gridDim.x);
          next = 0;
        } else {
          next = c;  // there is none: the present one again
        }
        if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_flag, p.status, 6u)) { ok = false; break; }
        tc_fence_after();
        switch (how(next)) {
          case BY32: store_and_load(s, s_before, std::integral_constant<int, BY32>()); break;
          case BY16: store_and_load(s, s_before, std::integral_constant<int, BY16>()); break;
          case FLOATS: store_and_load(s, s_before, std::integral_constant<int, FLOATS>()); break;
          default: store_and_load(s, s_before, std::integral_constant<int, CHECKED>());
        }
        if (before_first) {  // nothing is under way that would hide the wait
          hand_over(s);
          before_first = false;
        } else {
          s_before = s;
        }
        if (++s == STAGES) { s = 0; phase ^= 1; }
      }
    }
    if (ok && s_before >= 0) hand_over(s_before);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(T_ALL) : "memory");
  }
}

int pieces(const void* p, long long ld) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  return at % 32 == 0 && ld % 8 == 0 ? 2 : at % 16 == 0 && ld % 4 == 0 ? 1 : 0;
}

int how_to_read(const GemmDesc& g) {
  const int a = g.sAk == 1 ? pieces(g.A, g.sAm) : BY32, b = pieces(g.B, g.sBk == 1 ? g.sBn : g.sBk);  // M contiguous: by floats anyway
  return a < b ? a : b;
}

template <bool AK, bool BK>
cudaError_t launch(const SplitParams& p, int sms, cudaStream_t stream) {
  static std::mutex attr_mutex;
  static unsigned long long attr_set = 0;  // one bit per device ordinal
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!(attr_set >> (dev & 63) & 1ull)) {
      cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<AK, BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
      if (e != cudaSuccess) return e;
      attr_set |= 1ull << (dev & 63);
    }
  }
  gemm_split_kernel<AK, BK><<<p.tiles < sms ? p.tiles : sms, SPLIT_THREADS, SMEM_BYTES, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace

// us: 6 and 0.88 per chunk and round of the tiles, 1.37 where rows are not whole 16-byte pieces.
double gemm_split_us(const GemmDesc& g, int sms) {
  const long long tiles = (long long)((g.M + 127) / 128) * ((g.N + BN - 1) / BN);
  const double rounds = (double)((tiles + sms - 1) / sms), chunks = (g.K + CHUNK_K - 1) / CHUNK_K;
  return 6.0 + rounds * chunks * (how_to_read(g) != FLOATS ? 0.88 : 1.37);
}

// By the estimates of both sides, fitted to 110 shapes of 16 to 4096 rows, columns and k in the three forms of the step (the
// faster one is missed by 2 % on average). Sums of fewer than 64 terms stay on the CUDA cores: neither faster here nor more
// precise.
bool gemm_split_serves(const GemmDesc& g, int sms) {
  if (g.in_type != T_F32 || g.out_type != T_F32 || g.M <= 16 || g.N <= 16 || g.K < 64) return false;
  if ((g.sAk != 1 && g.sAm != 1) || (g.sBk != 1 && g.sBn != 1)) return false;
  if ((long long)((g.M + 127) / 128) * ((g.N + BN - 1) / BN) > 1 << 30) return false;
  return gemm_split_us(g, sms) <= gemm_simt_us(g);
}

cudaError_t gemm_split_launch(const GemmDesc& g, int sms, cudaStream_t stream, unsigned int* status) {
  SplitParams p;
  p.g = g;
  p.how_ab = how_to_read(g);
  p.vec_c = pieces(g.C, g.ldc);
  p.vec_x = pieces(g.aux, g.ldaux);
  p.status = status;
  p.n_blocks = (g.N + BN - 1) / BN;
  p.tiles = (g.M + 127) / 128 * p.n_blocks;
  if (g.sAk == 1 && g.sBk == 1) return launch<true, true>(p, sms, stream);
  if (g.sAk == 1) return launch<true, false>(p, sms, stream);
  if (g.sBk == 1) return launch<false, true>(p, sms, stream);
  return launch<false, false>(p, sms, stream);
}

}  // namespace b2
