// A whole training step - or several - in one launch, for networks whose GEMMs are too small to fill
// the GPU for long.
//
// As one launch per GEMM such a step is a chain of 2L kernels (forward, then input gradients) of
// which each pays launch, pipeline fill, an exposed epilogue and drain before the next may start, with
// most SMs idle (a 1024 x 1024 layer is 64 tiles of 128 x 128). Here one persistent CTA per SM walks a
// fixed list of output tiles of all GEMMs of the step:
//
//   fwd(0) .. fwd(L-1), then for l = L-1 .. 0: dgrad(l) and, one or two layers behind, wgrad
//
// round-robin over the grid, and a tile starts as soon as the tiles that produce its operands are
// done: a forward or input-gradient tile waits for the row block it reads, a weight-gradient tile for
// the whole gradient matrix. So layers overlap row block by row block, and the weight gradients fill the
// SMs that the chain of input gradients leaves free. The element-wise kernels are gone: the epilogue of
// the last forward GEMM computes the output gradient and the loss, the epilogue of a weight-gradient
// tile updates the weights (after every input-gradient tile that reads them).
//
// Every tile waits only for tiles earlier in the list and every CTA takes its tiles in list order, so with
// all CTAs resident (cooperative launch, at most one per SM) some CTA can always proceed. All waits are
// bounded as in gemm_tc_kernel.
//
// Roles per CTA as in gemm_tc_kernel: warp 0 TMA producer (also waits for the dependencies), warp 1 MMA
// issuer, warps 2-9 epilogue in two groups of four; two TMEM accumulators. A stage holds two 128-byte slabs of K
// (one in the fp32-class mode): the issuing threads' instructions per stage bound these short k-loops. While a tile
// waits for the tiles that produce its A, its weights already fill the ring.
//
// Two forms: a CTA per tile (128 x 64 or 128 x 128), and CTA pairs (cta_group::2, 256 x 128, each CTA holds 128 rows of
// A and half of B) for networks whose layers fill the GPU.
//
// What bounds it: with a CTA per tile the latency of one layer after another. In-kernel stamps of a 1024 x 1024 layer at
// batch 1024, taken before the 32-byte stores: 1.1 us from "dependency met" to the first operands, 2.5 us for 16 k-blocks,
// 1.2 us epilogue (weight update 3.6 us, loss 3.3 us), 1.2 us until the stores are visible to the other SMs, 0.8 us until
// the next tile's producer has seen the counter. No unit is busy meanwhile (tensor pipe 16 %, L2 26 % of peak). The pair form
// has no counters: a cooperative launch of clusters does not replay under the profiler. Loops must not spill to local
// memory here: the acquiring loads of the counters drop the L1, and each reload is an L2 round trip (two spilling epilogue
// groups: 110 -> 135 us per step, without spills 97; what is left are 4 to 16 bytes in three of the six kernels).
// bf16, us per step, launch per GEMM -> here: 5 x 1024, batch 1024 170 -> 89; 20 x 512, batch 2048 589 -> 233;
// 784-500-300-10, batch 1000 87 -> 47; 6 x 512, batch 8192 -> 158 (pairs).
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "row_pieces.h"
#include "tcgen05.cuh"

namespace b2 {
namespace {

enum StepEpi : int { SE_NONE = 0, SE_RELU = 1, SE_MASK = 2, SE_LOSS = 3, SE_SGD = 4, SE_NARROW = 5 };
enum OpForm : int { OP_K2D = 0, OP_K3D = 1, OP_MN3D = 2, OP_MN2D = 3 };
constexpr int STEP_THREADS = 64 + 2 * 128;   // producer warp, MMA warp, two groups of four epilogue warps
constexpr int EPI_BYTES = 8 * 4096;          // a chunk buffer of 32 rows x 128 bytes per epilogue warp

// One operand of a GEMM: how its slabs are fetched and described to the tensor core.
struct Operand {
  int form, boxes;        // boxes: 128-byte columns per slab (OP_MN2D)
  uint32_t col_bytes;     // distance of those columns in shared memory
  uint32_t bytes;         // bytes of a stage taken by this operand (without its twin)
  uint32_t kstep16, slab16;  // descriptor advance per k-step and per 128-byte slab of K, in 16-byte units
  uint64_t desc;          // descriptor without its address
};
struct StepMaps {
  CUtensorMap a, b, c, a_lo, b_lo;  // c: output and weight gradients
};
struct StepOp {
  Operand a, b;
  int M, N, num_n, num_kb, block_n;
  int first_item;
  uint32_t idesc, tx_bytes;
  int epi, out_bf16, wide;          // wide: rows of the result start on 32-byte boundaries
  int ld;                           // row pitch of C and, element for element, of w, w16, w_lo, target, dz
  int ld_mask;
  uint32_t* mask_out;
  const uint32_t* mask_in;
  union {
    float* w;                       // weight update
    void* c;                        // hidden layer: result
  };
  __nv_bfloat16* w16;
  union {
    float* w_lo;
    float* c_lo;                    // low-order twin of the result
  };
  // What has to be finished before a tile may load: indices into the counters (-1: nothing) and the counts a
  // step adds to them (every epilogue warp of a tile adds one).
  int row_cnt, row_target;          // counter of row block 0 of the operand's producer
  int all_cnt, all_target;          // all tiles of the producer (weight gradient)
  int prev_cnt[2], prev_target[2];  // weight updates of the previous step: this layer's and the next one's
  union {
    int upd_cnt;                    // weight gradient: input gradient of the same layer (reads the old weights)
    int mask_cnt;                   // input gradient: row block 0 of the GEMM that writes mask_in
  };
  union { int upd_target, mask_target; };
  int sig_row, sig_all, own_target; // counters this op raises (-1: nobody waits for them)
};

constexpr int EARLY_POLLS = 1 << 16;  // polls (about 0.5 us each) of the loop that loads weights ahead of a dependency

struct StepHead {
  const StepMaps* maps;
  unsigned int* counters;
  unsigned int* status;
  int nops, items, steps;
  int stages;
  uint32_t slot_bytes;
  int tmem_cols;
  float neg_lr;
  // output gradient and loss
  int baseline;
  float inv_batch;
  const float* target;
  void* dz;
  float* dz_lo;
  double* loss;
  double loss_scale;
  // narrow last layer (SE_NARROW): activation, weights, result
  const void* nar_a;
  const void* nar_w;
  float* nar_y;
  int nar_k, nar_lda;
};
// The scalars travel as kernel parameters, in the constant bank: read from global memory they cost an L2
// round trip per cache line and tile, because every acquiring load of a counter drops the L1. So a step may
// have as many GEMMs as fit into the 32 764 bytes of parameters a launch can take, about 50 layers. Every launch
// copies its parameters, whatever part of them is used (3 small layers, one blocking step: 89 us with 32 KB
// against 77 us with 14 KB), so there is a smaller table for the usual depths, up to 21 layers.
constexpr int SMALL_OPS = 64;
constexpr int MAX_OPS = (int)((32764 - sizeof(StepHead)) / sizeof(StepOp));
template <int OPS>
struct StepArgs : StepHead {
  StepOp op[OPS];
};

__device__ __forceinline__ float lo_part(float v) {
  return v - __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
}

// Walks this CTA's items: step `it`, op `op`, item `w` of the step's list.
struct Walk {
  int w, it, op;
  __device__ __forceinline__ void begin(int unit) { w = unit; it = 0; op = 0; }
  template <int OPS>
  __device__ __forceinline__ bool settle(const StepArgs<OPS>& p) {
    while (w >= p.items) { w -= p.items; ++it; op = 0; }
    if (it >= p.steps) return false;
    while (op + 1 < p.nops && w >= p.op[op + 1].first_item) ++op;
    return true;
  }
  __device__ __forceinline__ void advance(int units) { w += units; }
};

__device__ __forceinline__ bool wait_counter(const unsigned int* c, unsigned int target, volatile int* abort_flag,
                                             unsigned int* status, unsigned int code) {
  if (ld_acquire_u32(c) >= target) return true;
  unsigned long long t0 = 0;
  unsigned int spins = 0;
  while (ld_acquire_u32(c) < target) {
    if ((++spins & 0xFF) == 0) {
      if (*abort_flag) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > WAIT_LIMIT_NS) {
        *abort_flag = 1;
        atomicCAS(status, 0u, code);
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void count_up(unsigned int* c) {  // after a fence
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
}

// A slab of K in the fp32-class mode: A*B, A*B_lo and A_lo*B as two MMAs per k-step. B and its twin lie one behind the
// other in the stage, so that A meets both as one operand of 2N columns (main sum | corrections): every MMA reads its
// operands from shared memory, which bounds this loop, and A is the larger one (128 x 64 tiles: 18 -> 14 KB per k-step).
// The terms enter each accumulator in the order of issue_ksteps.
__device__ __forceinline__ void issue_ksteps_x3(uint32_t tmem_d, uint64_t adesc0, uint64_t bdesc0, uint32_t a_step16,
                                                uint32_t b_step16, uint32_t idesc, int block_n, uint32_t accumulate0,
                                                uint32_t alo16) {
  const uint32_t idesc2 = idesc + ((uint32_t)(block_n >> 3) << 17);  // N is twice as large
#pragma unroll
  for (int ks = 0; ks < KSTEPS; ++ks) {
    const uint64_t a = adesc0 + (uint64_t)(ks * a_step16), b = bdesc0 + (uint64_t)(ks * b_step16);
    mma_issue<true, false>(tmem_d, a, b, idesc2, ks == 0 ? accumulate0 : 1u);
    mma_issue<true, false>(tmem_d + (uint32_t)block_n, a + (uint64_t)alo16, b, idesc, 1u);
  }
}

template <int SLABS, bool PAIR>
__device__ __forceinline__ void load_operand(const Operand& o, const CUtensorMap* map, uint32_t bar, uint32_t dst,
                                             int kb, int slab_k, int mn0, int col_log2) {
  const int k0 = kb * SLABS * slab_k;
  if (o.form == OP_K3D) {
    tma_load_3d<PAIR>(map, bar, dst, 0, mn0, kb * SLABS);
  } else if (o.form == OP_MN3D) {
    tma_load_3d<PAIR>(map, bar, dst, 0, k0, mn0 >> col_log2);
  } else if (o.form == OP_K2D) {
#pragma unroll
    for (int s = 0; s < SLABS; ++s)
      tma_load_2d<PAIR>(map, bar, dst + (uint32_t)s * (o.bytes / SLABS), k0 + s * slab_k, mn0);
  } else {
    for (int c = 0; c < o.boxes; ++c)
      tma_load_2d<PAIR>(map, bar, dst + (uint32_t)c * o.col_bytes, mn0 + (c << col_log2), k0);
  }
}

// Output gradient and loss of four consecutive columns (loss_grad_kernel's arithmetic); t = targets.
template <bool BF16>
__device__ __forceinline__ float loss_piece(const StepHead& p, size_t at, const uint4& v, const float4& t) {
  float4 d = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
  float4 g = d;
  if (p.baseline) {
    d.x -= t.x; d.y -= t.y; d.z -= t.z; d.w -= t.w;
    g.x = d.x * p.inv_batch; g.y = d.y * p.inv_batch; g.z = d.z * p.inv_batch; g.w = d.w * p.inv_batch;
  }
  if (BF16) {
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.dz) + at) =
        make_uint2(pack_bf16(g.x, g.y), pack_bf16(g.z, g.w));
  } else {
    *reinterpret_cast<float4*>(static_cast<float*>(p.dz) + at) = g;
    if (p.dz_lo)
      *reinterpret_cast<float4*>(p.dz_lo + at) = make_float4(lo_part(g.x), lo_part(g.y), lo_part(g.z), lo_part(g.w));
  }
  return 0.5f * (d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w);
}

// w = fma(-lr, g, w) for four consecutive columns (sgd_kernel's arithmetic).
__device__ __forceinline__ float4 sgd4(float4 w, float g0, float g1, float g2, float g3, float neg_lr) {
  return make_float4(fmaf(neg_lr, g0, w.x), fmaf(neg_lr, g1, w.y), fmaf(neg_lr, g2, w.z), fmaf(neg_lr, g3, w.w));
}
__device__ __forceinline__ void sgd_store(const StepOp& o, size_t at, float4 v) {
  *reinterpret_cast<float4*>(o.w + at) = v;
  if (o.w16) *reinterpret_cast<uint2*>(o.w16 + at) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  if (o.w_lo)
    *reinterpret_cast<float4*>(o.w_lo + at) = make_float4(lo_part(v.x), lo_part(v.y), lo_part(v.z), lo_part(v.w));
}
// 32 bytes of a row to global memory: one store where rows start on 32-byte boundaries, else a 16-byte piece at a time
// (`pieces` = how many of the two lie in the matrix, 0 to 2). A row per lane: a 16-byte store is half a sector. us per
// step, all as 16-byte pieces -> 32 bytes: 20 x 512, batch 2048 bf16 243 -> 234, fp32-class 592 -> 577; as pairs 6 x 512,
// batch 8192 bf16 165 -> 159, tf32 262 -> 247, fp32-class 500 -> 467; 5 x 1024, batch 1024 bf16 91 -> 89.
__device__ __forceinline__ void store32(void* at, const uint32_t* r, bool wide, int pieces) {
  if (wide && pieces == 2) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
    return;
  }
  if (pieces > 0) *reinterpret_cast<uint4*>(at) = make_uint4(r[0], r[1], r[2], r[3]);
  if (pieces > 1) *(reinterpret_cast<uint4*>(at) + 1) = make_uint4(r[4], r[5], r[6], r[7]);
}

// 16-byte piece `piece` of row `row` of a chunk (128-byte swizzle).
__device__ __forceinline__ const uint8_t* chunk_piece(const uint8_t* chunk, int row, int piece) {
  return chunk + row * 128 + ((piece ^ (row & 7)) << 4);
}
// at += step, opaque to the compiler, which would otherwise hold the addresses of all eight rows at once
__device__ __forceinline__ void step_row(size_t& at, size_t step) {
  at += step;
  asm volatile("" : "+l"(at));
}

// The fp32 values (weights or targets) that belong to a chunk of 32 rows x 32 columns, in the order in which
// the element-wise part of the epilogue takes the chunk's pieces: lanes 8i .. 8i+7 cover one row.
__device__ __forceinline__ void load_chunk(float4 (&v)[8], const float* base, size_t ld, int row0, int M, int gcol, int N,
                                           int lane) {
  const int rows = gcol < N ? M - row0 - (lane >> 3) : 0;
  size_t at = (size_t)(row0 + (lane >> 3)) * ld + gcol;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = 4 * i < rows ? __ldcg(reinterpret_cast<const float4*>(base + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
    step_row(at, 4 * ld);
  }
}

// Eight consecutive elements of a bf16 row, four of an fp32 row, the 16 bytes masked by `m` (the padding behind the
// last column may hold NaNs). Written by other SMs during this launch: read past the L1.
template <bool BF16>
__device__ __forceinline__ uint4 load_row_piece(const void* row, int k, const uint32_t (&m)[4]) {
  if (!BF16) return __ldcg(reinterpret_cast<const uint4*>(static_cast<const float*>(row) + k));  // rows of whole pieces
  const uint4 u = __ldcg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(row) + k));
  return make_uint4(u.x & m[0], u.y & m[1], u.z & m[2], u.w & m[3]);
}
template <bool BF16>
__device__ __forceinline__ float row_elem(const uint4& u, int i) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  if (!BF16) return __uint_as_float(w[i & 3]);
  return __uint_as_float(i & 1 ? w[i >> 1] & 0xFFFF0000u : w[i >> 1] << 16);
}

// Last layer with fewer than 16 outputs, too narrow for a tensor-core tile: two rows per epilogue warp on the
// CUDA cores, lanes split K. The weight rows come eight at a time, all loads before the first use: one at a time the
// L2's latency per row added up (10 outputs of 300: 75 us). Returns this lane's share of the loss.
constexpr int NARROW_R = 2, NARROW_ROWS = 4 * NARROW_R;  // rows of a warp and of an item
constexpr int NARROW_ITEMS = BLOCK_M / NARROW_ROWS;         // items of a row block, of one CTA or of a pair
template <bool BF16, int NMAX>
__device__ __forceinline__ float narrow_rows(const StepHead& p, int row0, int M, int N, int ld, int lane) {
  constexpr int V = BF16 ? 8 : 4, R = NARROW_R, NB = NMAX < 8 ? NMAX : 8;
  const size_t row_bytes = (size_t)p.nar_lda * (BF16 ? 2 : 4);
  float loss = 0.f;
  if (row0 >= M) return loss;
  float acc[R][NMAX];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int n = 0; n < NMAX; ++n) acc[r][n] = 0.f;
  for (int k = lane * V; k < p.nar_k; k += 32 * V) {
    uint32_t m[4];  // bf16: which halves of the piece lie in front of column K
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int left = p.nar_k - k - 2 * i;
      m[i] = left > 1 ? 0xFFFFFFFFu : left == 1 ? 0xFFFFu : 0u;
    }
    uint4 a[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      a[r] = load_row_piece<BF16>(static_cast<const char*>(p.nar_a) + (size_t)min(row0 + r, M - 1) * row_bytes, k, m);
#pragma unroll
    for (int n0 = 0; n0 < NMAX; n0 += NB) {
      if (n0 >= N) break;
      uint4 b[NB];
#pragma unroll
      for (int n = 0; n < NB; ++n)
        b[n] = load_row_piece<BF16>(static_cast<const char*>(p.nar_w) + (size_t)min(n0 + n, N - 1) * row_bytes, k, m);
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int i = 0; i < V; ++i)
            acc[r][n0 + n] = fmaf(row_elem<BF16>(a[r], i), row_elem<BF16>(b[n], i), acc[r][n0 + n]);
    }
  }
#pragma unroll
  for (int n = 0; n < NMAX; ++n) {
    if (n >= N) break;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r][n] += __shfl_xor_sync(0xFFFFFFFFu, acc[r][n], s);
    float y = acc[0][n];  // lane r finishes row r
#pragma unroll
    for (int r = 1; r < R; ++r) y = lane == r ? acc[r][n] : y;
    const int row = row0 + lane;
    if (lane < R && row < M) {
      const size_t at = (size_t)row * ld + n;
      p.nar_y[at] = y;
      const float d = p.baseline ? y - __ldg(p.target + at) : y;
      const float gr = p.baseline ? d * p.inv_batch : y;
      if (BF16) {
        static_cast<__nv_bfloat16*>(p.dz)[at] = __float2bfloat16_rn(gr);
      } else {
        static_cast<float*>(p.dz)[at] = gr;
        if (p.dz_lo) p.dz_lo[at] = lo_part(gr);
      }
      loss += 0.5f * d * d;
    }
  }
  return loss;
}

template <int KIND, int OPS, bool PAIR>
__global__ void __launch_bounds__(STEP_THREADS, 1) step_kernel(const __grid_constant__ StepArgs<OPS> p) {
  constexpr bool TF32 = KIND != KIND_BF16, X3 = KIND == KIND_X3;
  constexpr int SLABS = X3 ? 1 : 2;
  constexpr int ROWS = PAIR ? 2 * BLOCK_M : BLOCK_M;  // rows of a tile
  constexpr int SLAB_K = TF32 ? 32 : 64, COL_LOG2 = TF32 ? 5 : 6;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full_bar[2];
  __shared__ __align__(8) uint64_t acc_empty_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_s;
  const int rank = PAIR ? (int)cluster_ctarank() : 0;
  const int unit = PAIR ? blockIdx.x >> 1 : blockIdx.x, units = PAIR ? gridDim.x >> 1 : gridDim.x;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full_bar[a], 1);
      mbar_init(&acc_empty_bar[a], PAIR ? 16 : 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                   "r"((uint32_t)p.tmem_cols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                   "r"((uint32_t)p.tmem_cols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // no remote arrival before the barriers exist
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  // TMEM columns of one accumulator (fp32-class: with its corrections behind it, of a pair behind both accumulators)
  const uint32_t acc_cols = X3 && PAIR ? 128u : (uint32_t)p.tmem_cols / 2;
  Walk wk;
  wk.begin(unit);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t full_own = smem_u32(full_bar), empty0 = smem_u32(empty_bar), ring0 = smem_u32(smem);
      const uint32_t full0 = PAIR ? map_to_cta(full_own, 0) : full_own;  // the leader's counts the bytes of both CTAs
      const int stages = p.stages;
      const uint32_t slot = p.slot_bytes;
      while (ok && wk.settle(p)) {
        const StepOp& o = p.op[wk.op];
        if (o.epi == SE_NARROW) { wk.advance(units); continue; }
        const StepMaps* mp = p.maps + wk.op;
        asm volatile("prefetch.tensormap [%0];" ::"l"(&mp->a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&mp->b) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&mp->c) : "memory");
        const int idx = wk.w - o.first_item;
        const int num_n = o.num_n, nkb = o.num_kb;
        const int mb = idx / num_n, nb = idx - mb * num_n;
        const int m0 = mb * ROWS + rank * BLOCK_M;                        // this CTA's rows of A
        const int n0 = nb * o.block_n + (PAIR ? rank * (o.block_n >> 1) : 0);  // and of B
        const uint32_t tx = o.tx_bytes * (PAIR ? 2u : 1u);
        const Operand oa = o.a, ob = o.b;
        const uint32_t a_bytes = oa.bytes, b_bytes = ob.bytes;
        const unsigned int it = (unsigned int)wk.it;
        if (it > 0) {
          // weights updated by the previous step; with them all readers of the buffers this tile overwrites are done
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (ok && o.prev_cnt[i] >= 0)
              ok = wait_counter(p.counters + o.prev_cnt[i], it * (unsigned int)o.prev_target[i], abort_flag, p.status, 8u);
        }
        int early = 0;  // stages whose B slabs are on their way before A exists
        int estage = stage;
        uint32_t ephase = phase;
        int polls = 0;
        if (ok && o.row_cnt >= 0) {
          // B holds weights: while the tiles that produce A are computed, its slabs may already fill the ring
          const unsigned int target = (it + 1) * (unsigned int)o.row_target;
          const unsigned int* const cnt = p.counters + o.row_cnt + mb;
          const int most = min(stages, nkb);
          if (it > 0) fence_proxy_async_all();
          while (early < most && ld_acquire_u32(cnt) < target) {
            if (!mbar_test_wait(empty0 + 8u * estage, ephase ^ 1)) {
              if (++polls > EARLY_POLLS) break;  // the bounded waits below take over
              continue;
            }
            const uint32_t full = full0 + 8u * estage;
            const uint32_t sb = ring0 + (uint32_t)estage * slot + a_bytes * (X3 ? 2u : 1u);
            if (rank == 0) mbar_expect_tx(full_own + 8u * estage, tx);
            load_operand<SLABS, PAIR>(ob, &mp->b, full, sb, early, SLAB_K, n0, COL_LOG2);
            if (X3) load_operand<SLABS, PAIR>(ob, &mp->b_lo, full, sb + b_bytes, early, SLAB_K, n0, COL_LOG2);
            ++early;
            if (++estage == stages) { estage = 0; ephase ^= 1; }
          }
          ok = wait_counter(cnt, target, abort_flag, p.status, 6u);
        }
        if (ok && o.all_cnt >= 0)
          ok = wait_counter(p.counters + o.all_cnt, (it + 1) * (unsigned int)o.all_target, abort_flag, p.status, 7u);
        if (!ok) break;
        fence_proxy_async_all();  // the acquired data is read through the async proxy next
        for (int kb = 0; kb < nkb; ++kb) {
          const uint32_t full = full0 + 8u * stage;
          const uint32_t sa = ring0 + (uint32_t)stage * slot;
          const uint32_t sb = sa + a_bytes * (X3 ? 2u : 1u);
          if (kb >= early) {
            if (!mbar_wait(empty0 + 8u * stage, phase ^ 1, abort_flag, p.status, 1u)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(full_own + 8u * stage, tx);
          }
          load_operand<SLABS, PAIR>(oa, &mp->a, full, sa, kb, SLAB_K, m0, COL_LOG2);
          if (X3) load_operand<SLABS, PAIR>(oa, &mp->a_lo, full, sa + a_bytes, kb, SLAB_K, m0, COL_LOG2);
          if (kb >= early) {
            load_operand<SLABS, PAIR>(ob, &mp->b, full, sb, kb, SLAB_K, n0, COL_LOG2);
            if (X3) load_operand<SLABS, PAIR>(ob, &mp->b_lo, full, sb + b_bytes, kb, SLAB_K, n0, COL_LOG2);
          }
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        wk.advance(units);
      }
      if (!ok) {  // give copies already in flight a bounded time to land before the CTA retires
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------- MMA issuer (of a pair: the leader's)
    if (rank == 0 && elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar), acc_full0 = smem_u32(acc_full_bar);
      const uint32_t ring16 = smem_u32(smem) >> 4, slot16 = p.slot_bytes >> 4;
      const int stages = p.stages;
      while (ok && wk.settle(p)) {
        const StepOp& o = p.op[wk.op];
        if (o.epi == SE_NARROW) { wk.advance(units); continue; }
        const int nkb = o.num_kb;
        const uint32_t idesc = o.idesc;
        const uint32_t a16 = o.a.bytes >> 4, b16 = o.b.bytes >> 4;
        const uint32_t a_step = o.a.kstep16, b_step = o.b.kstep16, a_slab = o.a.slab16, b_slab = o.b.slab16;
        const uint64_t a0 = o.a.desc + ring16, b0 = o.b.desc + ring16 + a16 * (X3 ? 2u : 1u);
        if (!mbar_wait(&acc_empty_bar[acc], acc_phase ^ 1, abort_flag, p.status, 2u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)acc * acc_cols;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(full0 + 8u * stage, phase, abort_flag, p.status, 3u)) { ok = false; break; }
          tc_fence_after();
          const uint32_t off = (uint32_t)stage * slot16;
#pragma unroll
          for (int s = 0; s < SLABS; ++s) {
            if (X3 && PAIR)
              issue_ksteps<1, true, true, true, KSTEPS>(tmem_d, a0 + off, b0 + off, a_step, b_step, idesc, 0u,
                                                        kb == 0 ? 0u : 1u, 0u, a16, b16);
            else if (X3)
              issue_ksteps_x3(tmem_d, a0 + off, b0 + off, a_step, b_step, idesc, o.block_n, kb == 0 ? 0u : 1u, a16);
            else
              issue_ksteps<1, TF32, PAIR, false, KSTEPS>(tmem_d, a0 + off + s * a_slab, b0 + off + s * b_slab, a_step,
                                                          b_step, idesc, 0u, (s == 0 && kb == 0) ? 0u : 1u, 0u, 0u, 0u);
          }
          if (PAIR) tc_commit_pair(empty0 + 8u * stage); else tc_commit(empty0 + 8u * stage);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (PAIR) tc_commit_pair(acc_full0 + 8u * acc); else tc_commit(acc_full0 + 8u * acc);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        wk.advance(units);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    // One CTA: a group takes every other tile, those in TMEM accumulator `group`, so that an input gradient does not wait
    // behind the long epilogue of a weight gradient. A pair has half as many tiles, twice as large: a group takes half of
    // the columns of each.
    const int group = (warp - 2) >> 2;
    int acc = PAIR ? 0 : group;
    uint32_t acc_phase = 0;
    int turn = 0, narrow_turn = 0;
    const auto free_acc = [&]() {  // last read of the accumulator: the next tile may have it
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_leader(map_to_cta(smem_u32(&acc_empty_bar[acc]), 0));
        else mbar_arrive(&acc_empty_bar[acc]);
      }
    };
    const auto next_acc = [&]() {
      if (PAIR) acc ^= 1;
      if (!PAIR || acc == 0) acc_phase ^= 1;
    };
    uint8_t* const cbuf = smem + (size_t)p.stages * p.slot_bytes + (size_t)(warp - 2) * 4096;
    const uint32_t swz = (uint32_t)(lane & 7);
    // the loss reported is the last step's
    auto add_loss = [&](float loss) {
      double sum = (double)loss;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, s);
      if (lane == 0) atomicAdd(p.loss, sum * p.loss_scale);
    };
    // this warp's part of a tile is stored: complete the stores, then the counters
    auto publish = [&](int sig_row, int sig_all, bool bulk) {
      __syncwarp();
      if (lane == 0) {
        if (bulk) {
          bulk_wait_all();
          fence_proxy_async_all();
        }
        __threadfence();  // one fence for both counters
        if (sig_row >= 0) count_up(p.counters + sig_row);
        if (sig_all >= 0) count_up(p.counters + sig_all);
      }
    };
    while (wk.settle(p)) {
      const StepOp& o = p.op[wk.op];
      const int idx = wk.w - o.first_item;
      const int num_n = o.num_n, M = o.M, N = o.N, epi = o.epi;
      if (!PAIR || epi == SE_NARROW) {
        int& t = epi == SE_NARROW ? narrow_turn : turn;
        const bool mine = t == group;
        t ^= 1;
        if (!mine) { wk.advance(units); continue; }
      }
      if (epi == SE_NARROW) {  // an item is NARROW_ROWS rows here
        const int block = idx / NARROW_ITEMS;
        bool ok = o.row_cnt < 0 || wait_counter(p.counters + o.row_cnt + block, (wk.it + 1u) * o.row_target,
                                                abort_flag, p.status, 6u);
        if (ok && wk.it > 0 && o.prev_cnt[0] >= 0)
          ok = wait_counter(p.counters + o.prev_cnt[0], (unsigned int)wk.it * o.prev_target[0], abort_flag, p.status, 8u);
        if (!__all_sync(0xFFFFFFFFu, ok)) break;
        const int r0 = block * ROWS + rank * BLOCK_M + (idx - block * NARROW_ITEMS) * NARROW_ROWS + ((warp - 2) & 3) * NARROW_R;
        const float part = N <= 4 ? narrow_rows<!TF32, 4>(p, r0, M, N, o.ld, lane) : narrow_rows<!TF32, 16>(p, r0, M, N, o.ld, lane);
        if (wk.it + 1 == p.steps) add_loss(part);
        publish(o.sig_row >= 0 ? o.sig_row + block : -1, o.sig_all, true);
        wk.advance(units);
        continue;
      }
      const int mb = idx / num_n, nb = idx - mb * num_n;
      const int row0 = mb * ROWS + rank * BLOCK_M + q * 32, row = row0 + lane;
      const int width = PAIR ? o.block_n >> 1 : o.block_n, part0 = PAIR ? group * width : 0;  // this group's columns
      const int n0 = nb * o.block_n + part0;
      const bool out_bf16 = o.out_bf16 != 0;
      const size_t ld = (size_t)o.ld;
      const unsigned int it = (unsigned int)wk.it;
      if (epi < SE_LOSS) {
        // A hidden layer's result goes straight from registers to global memory, a row per lane. Through shared
        // memory and a TMA store the chain of layers paid 1.2 us to stage a tile and 1.8 us until it was visible.
        uint32_t mask[4] = {0, 0, 0, 0};
        bool ok = true;
        if (epi == SE_MASK) {  // written by other SMs during this launch: after their counter, and past the L1
          ok = wait_counter(p.counters + o.mask_cnt + mb, (it + 1) * (unsigned int)o.mask_target, abort_flag, p.status, 11u);
          const uint32_t* const m = o.mask_in + (long long)row * o.ld_mask + (n0 >> 5);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (ok && row < M && 32 * j < width && n0 + 32 * j < N) mask[j] = __ldcg(m + j);
        }
        ok = ok && mbar_wait(&acc_full_bar[acc], acc_phase, abort_flag, p.status, 4u);
        if (!__all_sync(0xFFFFFFFFu, ok)) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)acc * acc_cols + (uint32_t)part0;
        const bool wide = o.wide != 0;
        const int cols = min(width, N - n0);
        if (PAIR && cols <= 0) free_acc();
        uint32_t bits = 0;
#pragma unroll 1
        for (int c = 0; c < cols; c += 32) {
          uint32_t r[32];
          tmem_ld32(taddr + (uint32_t)c, r);
          if (X3) {
            uint32_t r2[32];
            tmem_ld32(taddr + (PAIR ? X3_CORR_COLS : (uint32_t)o.block_n) + (uint32_t)c, r2);
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
          }
          if (c + 32 >= cols) free_acc();
          if (epi == SE_RELU) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(fmaxf(__uint_as_float(r[j]), 0.f));
          } else if (epi == SE_MASK) {
            const uint32_t mk = c < 64 ? (c < 32 ? mask[0] : mask[1]) : (c < 96 ? mask[2] : mask[3]);
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = (mk >> j) & 1u ? r[j] : 0u;
          }
          uint32_t part[4] = {0, 0, 0, 0};
          const size_t at = (size_t)row * ld + n0 + c;
          if (out_bf16) {
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
            if (epi == SE_RELU) {  // bit = the stored half is non-zero (it is not negative)
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const uint32_t m = ((r[j] & 0x7FFF7FFFu) + 0x7FFF7FFFu) & 0x80008000u;
                part[j & 3] |= (((m >> 15) | (m >> 30)) & 3u) << (2 * j);
              }
            }
            if (row < M) {
              __nv_bfloat16* const dst = static_cast<__nv_bfloat16*>(o.c) + at;
#pragma unroll
              for (int j = 0; j < 2; ++j) store32(dst + 16 * j, r + 8 * j, wide, pieces_of_32(cols - c - 16 * j, 8));
            }
          } else {
            if (epi == SE_RELU) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (__uint_as_float(r[j]) > 0.f) part[j & 3] |= 1u << j;
            }
            if (row < M) {
              float* const dst = static_cast<float*>(o.c) + at;
#pragma unroll
              for (int j = 0; j < 4; ++j) store32(dst + 8 * j, r + 8 * j, wide, pieces_of_32(cols - c - 8 * j, 4));
              if (X3 && o.c_lo) {  // the low-order twin
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(lo_part(__uint_as_float(r[j])));
#pragma unroll
                for (int j = 0; j < 4; ++j) store32(o.c_lo + at + 8 * j, r + 8 * j, wide, pieces_of_32(cols - c - 8 * j, 4));
              }
            }
          }
          if (epi == SE_RELU && o.mask_out) {
            const uint32_t b = (part[0] | part[1]) | (part[2] | part[3]);
            uint32_t* const m = o.mask_out + (long long)row * o.ld_mask + ((n0 + c) >> 5);
            const bool odd = (c & 32) != 0;
            if (row < M) {  // two words at a time where that is an aligned pair
              if (o.ld_mask & 1) *m = b;
              else if (odd) *reinterpret_cast<uint2*>(m - 1) = make_uint2(bits, b);
              else if (c + 32 >= cols) *m = b;
            }
            bits = b;
          }
        }
        publish(o.sig_row >= 0 ? o.sig_row + mb : -1, o.sig_all, false);
        next_acc();
        wk.advance(units);
        continue;
      }
      const int chunk_cols = out_bf16 ? 64 : 32;  // 128 bytes of C per row and chunk
      const int nchunks = width / chunk_cols;
      const StepMaps* mp = p.maps + wk.op;
      const int piece = lane & 7;  // 16-byte piece of a row this lane takes in the element-wise part
      float loss = 0.f;
      const float* const extra = epi == SE_SGD ? o.w : p.baseline ? p.target : nullptr;
      const bool fetch = extra && !out_bf16;
      float4 pre[8];  // weights or targets of the next chunk, on their way while the MMAs run
      bool ok = true;
      if (epi == SE_SGD && it > 0)  // the update of the step before, possibly by another SM
        ok = wait_counter(p.counters + o.sig_all, it * (unsigned int)o.own_target, abort_flag, p.status, 10u);
      if (fetch) load_chunk(pre, extra, ld, row0, M, n0 + piece * 4, N, lane);
      if (ok && epi == SE_SGD && o.upd_cnt >= 0)
        ok = wait_counter(p.counters + o.upd_cnt, (it + 1) * (unsigned int)o.upd_target, abort_flag, p.status, 9u);
      ok = ok && mbar_wait(&acc_full_bar[acc], acc_phase, abort_flag, p.status, 4u);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)acc * acc_cols + (uint32_t)part0;
      if (PAIR && n0 >= N) free_acc();
      for (int ch = 0; ch < nchunks; ++ch) {
        const int col0 = n0 + ch * chunk_cols;
        if (col0 >= N) break;  // uniform across the warp
        const bool last = (ch == nchunks - 1) || (col0 + chunk_cols >= N);
        uint8_t* const dst = cbuf + (size_t)lane * 128;
        uint32_t r[32];
        // 32 columns at a time, and no more of them in registers than those: a value spilled to local memory costs
        // a round trip to the L2 here, because every acquiring load of a counter drops the L1
#pragma unroll 1
        for (int half = 0; half < (out_bf16 ? 2 : 1); ++half) {
          const uint32_t tcol = taddr + (uint32_t)(ch * chunk_cols + half * 32);
          tmem_ld32(tcol, r);
          if (X3) {
            uint32_t r2[32];
            tmem_ld32(tcol + (PAIR ? X3_CORR_COLS : (uint32_t)o.block_n), r2);
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
          }
          if (last && (half == 1 || !out_bf16)) free_acc();
          if (half == 0) {
            if (lane == 0) bulk_wait_read<0>();  // the store before has read the buffer
            __syncwarp();
          }
          if (out_bf16) {
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
            const uint32_t piece0 = (uint32_t)half << 2;
#pragma unroll
            for (int j = 0; j < 4; ++j)  // 128-byte swizzle: piece j of row `lane` at slot j ^ (lane & 7)
              *reinterpret_cast<uint4*>(dst + (((piece0 + j) ^ swz) << 4)) =
                  make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(dst + ((j ^ swz) << 4)) =
                  make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < M) {
          tma_store_2d(&mp->c, cbuf, col0, row0);
          bulk_commit();
        }
        {
          // element-wise work on the finished chunk, read back so that a warp instruction covers four whole
          // 128-byte rows: lanes 8i .. 8i+7 take the 16-byte pieces of one row
          const int gcol = col0 + piece * (out_bf16 ? 8 : 4);
          if (!out_bf16) {
            // behind the last column, in the row padding, an accumulator is 0 * operand: NaN after an Inf or a NaN
            const uint32_t m1 = gcol + 1 < N ? ~0u : 0u, m2 = gcol + 2 < N ? ~0u : 0u, m3 = gcol + 3 < N ? ~0u : 0u;
            const int rows = gcol < N ? M - row0 - (lane >> 3) : 0;  // row 4 * i of this lane's is inside if 4 * i < rows
            size_t at = (size_t)(row0 + (lane >> 3)) * ld + gcol;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint4 v = *reinterpret_cast<const uint4*>(chunk_piece(cbuf, 4 * i + (lane >> 3), piece));
              if (4 * i < rows) {
                if (epi == SE_LOSS)
                  loss += loss_piece<!TF32>(p, at, make_uint4(v.x, v.y & m1, v.z & m2, v.w & m3), pre[i]);
                else
                  sgd_store(o, at,
                            sgd4(pre[i], __uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z),
                                 __uint_as_float(v.w), p.neg_lr));
              }
              step_row(at, 4 * ld);
            }
            if (fetch && !last) load_chunk(pre, extra, ld, row0, M, gcol + 32, N, lane);
          } else {  // bf16 gradients: the update uses the stored (rounded) values
            const int rows = gcol < N ? M - row0 - (lane >> 3) : 0;
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
              load_chunk(pre, o.w + 4 * e, ld, row0, M, gcol, N, lane);
              size_t at = (size_t)(row0 + (lane >> 3)) * ld + gcol + 4 * e;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint2 v = *reinterpret_cast<const uint2*>(chunk_piece(cbuf, 4 * i + (lane >> 3), piece) + 8 * e);
                if (4 * i < rows)
                  sgd_store(o, at,
                            sgd4(pre[i], __uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u),
                                 __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u), p.neg_lr));
                step_row(at, 4 * ld);
              }
            }
          }
          __syncwarp();  // the next chunk overwrites what other lanes read
        }
      }
      if (epi == SE_LOSS && it + 1 == (unsigned int)p.steps) add_loss(loss);
      publish(o.sig_row >= 0 ? o.sig_row + mb : -1, o.sig_all, true);
      next_acc();
      wk.advance(units);
    }
    if (lane == 0) bulk_wait_all();
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // both CTAs are done with each other's shared memory and TMEM
  if (warp == 1) {
    tc_fence_after();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols)
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols)
                   : "memory");
  }
}

// ------------------------------------------------------------------ host side

// Tensor map of `dims` (innermost contiguous) with the 128-byte swizzle (atom32: in 32-byte atoms).
bool encode(CUtensorMap* map, const void* base, int eb, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
            const cuuint32_t* box, bool atom32, bool store) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, eb == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank,
             const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             atom32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
             store ? CU_TENSOR_MAP_L2_PROMOTION_NONE : CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// mn x k operand with `rows` of M or N per tile. One 3-D box per stage where the extents are whole
// 128-byte columns (K for a K-contiguous operand, M/N otherwise), else 2-D boxes.
bool make_operand(Operand& o, CUtensorMap& map, CUtensorMap& map_lo, const void* base, const void* lo, int eb,
                  long long mn, long long k, long long ld, bool mn_major, int rows, int slabs) {
  const int col = SLAB_BYTES / eb;
  const cuuint64_t pitch = (cuuint64_t)ld * eb;
  memset(&o, 0, sizeof o);
  o.bytes = (uint32_t)rows * SLAB_BYTES * slabs;
  auto both = [&](int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box, bool atom32) {
    if (!encode(&map, base, eb, rank, dims, strides, box, atom32, false)) return false;
    if (!lo) { map_lo = map; return true; }
    return encode(&map_lo, lo, eb, rank, dims, strides, box, atom32, false);
  };
  auto desc = [](uint32_t lbo, uint32_t sbo, uint32_t layout) {
    return ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)layout << 61);
  };
  if (!mn_major) {
    o.desc = desc(16, 8 * SLAB_BYTES, 2);
    o.kstep16 = KSTEP_BYTES >> 4;
    o.slab16 = (uint32_t)(rows * SLAB_BYTES) >> 4;
    if (k % col == 0) {
      const cuuint64_t dims[3] = {(cuuint64_t)col, (cuuint64_t)mn, (cuuint64_t)(k / col)};
      const cuuint64_t strides[2] = {pitch, SLAB_BYTES};
      const cuuint32_t box[3] = {(cuuint32_t)col, (cuuint32_t)rows, (cuuint32_t)slabs};
      o.form = OP_K3D;
      if (both(3, dims, strides, box, false)) return true;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)mn};
    const cuuint32_t box[2] = {(cuuint32_t)col, (cuuint32_t)rows};
    o.form = OP_K2D;
    return both(2, dims, &pitch, box, false);
  }
  const bool atom32 = eb == 4;  // 32-bit M/N-contiguous operands: the swizzle of 32-byte atoms
  const int block_k = slabs * col;
  o.boxes = rows / col;
  o.col_bytes = (uint32_t)block_k * SLAB_BYTES;
  o.desc = desc(o.col_bytes, atom32 ? 512 : 1024, atom32 ? 1 : 2);
  o.kstep16 = (uint32_t)((KSTEP_BYTES / eb) * SLAB_BYTES) >> 4;
  o.slab16 = KSTEPS * o.kstep16;
  if (mn % col == 0) {
    const cuuint64_t dims[3] = {(cuuint64_t)col, (cuuint64_t)k, (cuuint64_t)(mn / col)};
    const cuuint64_t strides[2] = {pitch, SLAB_BYTES};
    const cuuint32_t box[3] = {(cuuint32_t)col, (cuuint32_t)block_k, (cuuint32_t)o.boxes};
    o.form = OP_MN3D;
    if (both(3, dims, strides, box, atom32)) return true;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)mn, (cuuint64_t)k};
  const cuuint32_t box[2] = {(cuuint32_t)col, (cuuint32_t)block_k};
  o.form = OP_MN2D;
  return both(2, dims, &pitch, box, atom32);
}

}  // namespace

struct StepPlan {
  StepMaps* maps_dev = nullptr;
  int kind = KIND_BF16, grid = 0;
  bool pair = false;
  size_t smem = 0;
  StepArgs<MAX_OPS> args;  // counters, status, steps and learning rate are filled in per launch
};

template <int OPS>
using StepKernel = void (*)(const StepArgs<OPS>);
template <int OPS>
static cudaError_t pick_kernel(const StepPlan* plan, StepKernel<OPS>* kernel) {
  static const StepKernel<OPS> kernels[3][2] = {{step_kernel<KIND_BF16, OPS, false>, step_kernel<KIND_BF16, OPS, true>},
                                                {step_kernel<KIND_TF32, OPS, false>, step_kernel<KIND_TF32, OPS, true>},
                                                {step_kernel<KIND_X3, OPS, false>, step_kernel<KIND_X3, OPS, true>}};
  *kernel = kernels[plan->kind][plan->pair ? 1 : 0];
  // per launch: handles of several devices and threads share the library, and the call is cheap
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(*kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
}

template <int OPS>
static void launch_config(const StepPlan* plan, cudaStream_t stream, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[2]) {
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg->gridDim = dim3(plan->grid);
  cfg->blockDim = dim3(STEP_THREADS);
  cfg->dynamicSmemBytes = plan->smem;
  cfg->stream = stream;
  cfg->attrs = attr;
  cfg->numAttrs = plan->pair ? 2 : 1;
}

// Pairs that fit on the GPU at once: its SMs come in clusters that need not all hold whole pairs.
template <int OPS>
static int resident_pairs(const StepPlan* plan) {
  StepKernel<OPS> kernel;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  launch_config<OPS>(plan, nullptr, &cfg, attr);
  int n = 0;
  if (pick_kernel<OPS>(plan, &kernel) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(kernel), &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int step_plan_counters(const StepSpec& s) {
  int n = 0;
  for (const StepGemm& g : s.gemms) n += (g.d.M + BLOCK_M - 1) / BLOCK_M + 1;
  return n;
}

StepPlan* step_plan_create(const StepSpec& s, int sm_count) {
  const int nops = (int)s.gemms.size();
  if (nops < 1 || nops > MAX_OPS) return nullptr;
  const GemmDesc& d0 = s.gemms[0].d;
  const int eb = d0.in_type == T_BF16 ? 2 : 4;
  const bool x3 = d0.A_lo != nullptr;
  const int slabs = x3 ? 1 : 2;
  const bool pair = s.pair;
  const int rows = pair ? 2 * BLOCK_M : BLOCK_M;
  StepPlan* plan = new StepPlan();
  memset(&plan->args, 0, sizeof plan->args);
  StepArgs<MAX_OPS>& args = plan->args;
  StepOp* ops = args.op;
  std::vector<StepMaps> maps(nops);
  std::vector<int> row_base(nops), all_base(nops), ntiles(nops), per_item(nops), row_add(nops);
  std::vector<char> row_used(nops, 0), all_used(nops, 0);
  auto refuse = [&]() -> StepPlan* {
    step_plan_destroy(plan);
    return nullptr;
  };
  int ncnt = 0, items = 0, max_bn = 64;
  uint32_t slot = 0;
  for (int i = 0; i < nops; ++i) {
    const StepGemm& g = s.gemms[i];
    const GemmDesc& d = g.d;
    StepOp& o = ops[i];
    StepMaps& mp = maps[i];
    const int ob = d.out_type == T_BF16 ? 2 : 4;
    o.M = d.M; o.N = d.N;
    const int num_m = (d.M + rows - 1) / rows;
    o.block_n = g.block_n;
    o.num_n = (d.N + o.block_n - 1) / o.block_n;
    const int block_k = slabs * SLAB_BYTES / eb;
    o.num_kb = (d.K + block_k - 1) / block_k;
    const bool narrow = g.role == STEP_LAST_FWD && d.N < 16;
    if (narrow) {
      if (d.sAk != 1 || d.sBk != 1 || d.sAm != d.sBn || d.sAm % (16 / eb) != 0 || o.num_n != 1) return refuse();
      args.nar_a = d.A; args.nar_w = d.B; args.nar_y = static_cast<float*>(d.C);
      args.nar_k = d.K; args.nar_lda = (int)d.sAm;
    } else {
      const bool a_mn = d.sAm == 1 && d.sAk != 1, b_mn = d.sBn == 1 && d.sBk != 1;
      if (!make_operand(o.a, mp.a, mp.a_lo, d.A, d.A_lo, eb, d.M, d.K, a_mn ? d.sAk : d.sAm, a_mn, BLOCK_M, slabs) ||
          !make_operand(o.b, mp.b, mp.b_lo, d.B, d.B_lo, eb, d.N, d.K, b_mn ? d.sBk : d.sBn, b_mn,
                        pair ? o.block_n / 2 : o.block_n, slabs))
        return refuse();
      const cuuint64_t dims[2] = {(cuuint64_t)d.N, (cuuint64_t)d.M};
      const cuuint64_t pitch = (cuuint64_t)d.ldc * ob;
      const cuuint32_t box[2] = {(cuuint32_t)(128 / ob), 32};
      if (!encode(&mp.c, d.C, ob, 2, dims, &pitch, box, false, true)) return refuse();
      o.c = d.C;
      o.c_lo = static_cast<float*>(d.C_lo);
      o.wide = pitch % 32 == 0 && reinterpret_cast<uintptr_t>(d.C) % 32 == 0 && reinterpret_cast<uintptr_t>(d.C_lo) % 32 == 0;
      const uint32_t fmt = eb == 4 ? 2u : 1u;  // tf32 : bf16
      o.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
                ((uint32_t)(o.block_n >> 3) << 17) | ((uint32_t)(rows >> 4) << 24);
      o.tx_bytes = (o.a.bytes + o.b.bytes) * (x3 ? 2u : 1u);
      if (o.tx_bytes > slot) slot = o.tx_bytes;
      if (o.block_n > max_bn) max_bn = o.block_n;
    }
    o.out_bf16 = d.out_type == T_BF16;
    o.epi = narrow ? SE_NARROW : g.role == STEP_LAST_FWD ? SE_LOSS : g.role == STEP_WGRAD ? SE_SGD
            : d.epilogue == EPI_RELU ? SE_RELU : d.epilogue == EPI_MASK ? SE_MASK : SE_NONE;
    if (o.epi == SE_MASK && !g.mask_in) return refuse();
    o.mask_out = g.mask_out;
    o.mask_in = g.mask_in;
    o.ld_mask = (int)g.ld_mask;
    o.ld = (int)d.ldc;
    if (o.epi == SE_SGD) { o.w = g.w; o.w16 = g.w16; o.w_lo = g.w_lo; }
    o.first_item = items;
    ntiles[i] = narrow ? num_m * NARROW_ITEMS : num_m * o.num_n;
    // every epilogue warp counts one for each item it takes part in
    per_item[i] = pair ? (narrow ? 8 : 16) : 4;
    row_add[i] = per_item[i] * (narrow ? NARROW_ITEMS : o.num_n);
    items += ntiles[i];
    row_base[i] = ncnt;
    all_base[i] = ncnt + num_m;
    ncnt += num_m + 1;
  }
  for (int i = 0; i < nops; ++i) {
    const StepGemm& g = s.gemms[i];
    StepOp& o = ops[i];
    // a dependency always points to an earlier entry of the list, or to a weight gradient of the step before
    if (g.rows_of >= i || g.all_of >= i || g.update_after >= i || g.mask_of >= i) return refuse();
    o.row_cnt = g.rows_of >= 0 ? row_base[g.rows_of] : -1;
    o.row_target = g.rows_of >= 0 ? row_add[g.rows_of] : 0;
    o.all_cnt = g.all_of >= 0 ? all_base[g.all_of] : -1;
    o.all_target = g.all_of >= 0 ? per_item[g.all_of] * ntiles[g.all_of] : 0;
    o.upd_cnt = g.update_after >= 0 ? all_base[g.update_after] : -1;
    o.upd_target = g.update_after >= 0 ? per_item[g.update_after] * ntiles[g.update_after] : 0;
    for (int k = 0; k < 2; ++k) {
      o.prev_cnt[k] = g.prev_step[k] >= 0 ? all_base[g.prev_step[k]] : -1;
      o.prev_target[k] = g.prev_step[k] >= 0 ? per_item[g.prev_step[k]] * ntiles[g.prev_step[k]] : 0;
    }
    if (o.epi == SE_MASK) {
      if (g.mask_of < 0) return refuse();
      o.mask_cnt = row_base[g.mask_of];
      o.mask_target = row_add[g.mask_of];
      row_used[g.mask_of] = 1;
    }
    if (g.rows_of >= 0) row_used[g.rows_of] = 1;
    for (int j : {g.all_of, g.update_after, g.prev_step[0], g.prev_step[1], g.role == STEP_WGRAD ? i : -1})
      if (j >= 0) all_used[j] = 1;
  }
  for (int i = 0; i < nops; ++i) {
    ops[i].sig_row = row_used[i] ? row_base[i] : -1;
    ops[i].sig_all = all_used[i] ? all_base[i] : -1;
    ops[i].own_target = per_item[i] * ntiles[i];
  }
  plan->kind = x3 ? KIND_X3 : eb == 4 ? KIND_TF32 : KIND_BF16;
  args.nops = nops;
  args.items = items;
  args.slot_bytes = slot;
  plan->pair = pair;
  args.tmem_cols = x3 ? 512 : 2 * max_bn;
  args.target = s.target;
  args.dz = s.dz;
  args.dz_lo = s.dz_lo;
  args.baseline = s.baseline;
  args.inv_batch = s.inv_batch;
  args.loss_scale = s.loss_scale;
  args.loss = s.loss;
  const size_t budget = 227 * 1024 - 1024 /* alignment slack */ - 512 /* static: barriers */;
  args.stages = (int)((budget - EPI_BYTES) / slot);
  if (args.stages > MAX_STAGES) args.stages = MAX_STAGES;
  plan->smem = 1024 + (size_t)args.stages * slot + EPI_BYTES;
  if (plan->smem < 140 * 1024) plan->smem = 140 * 1024;  // one CTA (one TMEM allocation) per SM
  plan->grid = items < sm_count ? items : sm_count;
  if (pair) {
    int pairs = items < sm_count / 2 ? items : sm_count / 2;
    plan->grid = 2 * pairs;
    const int fit = nops <= SMALL_OPS ? resident_pairs<SMALL_OPS>(plan) : resident_pairs<MAX_OPS>(plan);
    if (fit < pairs) pairs = fit;
    if (pairs < 1) return refuse();
    plan->grid = 2 * pairs;
  }
  if (args.stages < 2 || cudaMalloc((void**)&plan->maps_dev, sizeof(StepMaps) * nops) != cudaSuccess ||
      cudaMemcpy(plan->maps_dev, maps.data(), sizeof(StepMaps) * nops, cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaGetLastError();
    return refuse();
  }
  args.maps = plan->maps_dev;
  return plan;
}

void step_plan_destroy(StepPlan* p) {
  if (!p) return;
  cudaFree(p->maps_dev);
  delete p;
}

template <int OPS>
static cudaError_t launch_ops(const StepPlan* plan, int steps, float lr, unsigned int* counters, unsigned int* status,
                              cudaStream_t stream) {
  StepKernel<OPS> kernel;
  cudaError_t e = pick_kernel<OPS>(plan, &kernel);
  if (e != cudaSuccess) return e;
  StepArgs<OPS> a;
  static_cast<StepHead&>(a) = plan->args;
  memcpy(a.op, plan->args.op, sizeof a.op);
  a.counters = counters;
  a.status = status;
  a.steps = steps;
  a.neg_lr = -lr;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  launch_config<OPS>(plan, stream, &cfg, attr);
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

cudaError_t step_launch(const StepPlan* plan, int steps, float lr, unsigned int* counters, unsigned int* status,
                        cudaStream_t stream) {
  return plan->args.nops <= SMALL_OPS ? launch_ops<SMALL_OPS>(plan, steps, lr, counters, status, stream)
                                      : launch_ops<MAX_OPS>(plan, steps, lr, counters, status, stream);
}

}  // namespace b2
