// Building blocks shared by the sm_100a tensor-core kernels (gemm_tcgen05.cu, step_kernel.cu): mbarriers, TMA
// loads and stores, tcgen05 MMA issue and TMEM reads as inline PTX, and the host's tensor maps.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace b2 {
namespace {

constexpr int BLOCK_M = 128;
constexpr int SLAB_BYTES = 128;          // bytes of the contiguous dimension per smem row
constexpr int KSTEP_BYTES = 32;          // bytes of K one tcgen05.mma consumes
constexpr int KSTEPS = SLAB_BYTES / KSTEP_BYTES;
constexpr int MAX_STAGES = 8;
constexpr int NUM_THREADS = 192;       // producer warp + MMA warp + 4 epilogue warps
constexpr int NUM_THREADS_SUB2 = 320;  // 256-row tiles: one group of 4 epilogue warps per 128-row accumulator
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;
enum MmaKind : int { KIND_BF16 = 0, KIND_TF32 = 1, KIND_X3 = 2 };
constexpr uint32_t X3_CORR_COLS = 256;  // fp32-class mode: TMEM column offset of the correction accumulators

// ------------------------------------------------------------------ PTX wrappers

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// One lane of a converged warp. The single-thread roles (TMA producer, MMA issuer) are entered through
// elect.sync and not through a test of the lane number: the compiler then knows that exactly one
// thread is active and feeds the descriptors and addresses of TMA and MMA instructions straight from
// uniform registers. Behind `if (lane == 0)` a k-block of four MMAs and one commit took 0.46 us to
// issue and one of two TMA loads 0.36 us, whatever the tile, and that was what bounded every GEMM
// (bf16, 8192 x 4096 x 4096 forward 212 -> 197 us, 512 x 512 x 2048 20.6 -> 16.5 us by this alone).
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {  // does not block
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false when it gave up or another role raised the abort flag. The timer is
// read only once in 256 failed polls: the waits of the pipeline are far shorter than that.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned int* status, unsigned int code) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = 0;
  unsigned int spins = 0;
  while (!mbar_try_wait(bar, parity)) {
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
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned int* status, unsigned int code) {
  return mbar_wait(smem_u32(bar), parity, abort_flag, status, code);
}
// TMA loads. `bar` is the shared-memory address of the barrier that counts the bytes; with PAIR
// (CTA-pair kernel) it is a shared::cluster address and may lie in the peer CTA. No multicast: the
// data lands in the issuing CTA's own shared memory only.
template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y) {
  if (PAIR)
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y, int z) {
  if (PAIR)
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// One operand slab of a k-block: `rows` elements of M or N from mn0 on, k-block starting at k0.
// K-contiguous storage: one box {block_k of K, rows}. M/N-contiguous storage: with `form` SLAB_MN3
// one 3-D box {128 bytes of M/N, block_k k-rows, 128-byte columns}, else (an extent of M or N that is
// not a whole number of 128-byte columns) one 2-D box per 128-byte column. The issuing thread's
// instructions bound short k-loops, so the number of boxes matters: with a box per column the
// weight gradient 512 x 512 x 2048 took 20.6 us against 16.5 us of the form with one box per slab.
enum SlabForm : int { SLAB_K = 0, SLAB_MN3 = 1, SLAB_MN2 = 2 };
template <bool PAIR>
__device__ __forceinline__ void load_slab(const CUtensorMap* map, uint32_t bar, uint32_t dst, int form, int k0, int mn0,
                                          int boxes, uint32_t box_bytes, int box_mn_log2) {
  if (form == SLAB_K) {
    tma_load_2d<PAIR>(map, bar, dst, k0, mn0);
  } else if (form == SLAB_MN3) {
    tma_load_3d<PAIR>(map, bar, dst, 0, k0, mn0 >> box_mn_log2);
  } else {
    for (int b = 0; b < boxes; ++b)
      tma_load_2d<PAIR>(map, bar, dst + (uint32_t)b * box_bytes, mn0 + (b << box_mn_log2), k0);
  }
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until at most N of this thread's bulk groups still READ their shared-memory source
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- CTA-pair (cta_group::2) forms
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of `local_addr` (a shared::cta address) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same for an arrival that orders no memory of this thread but its finished TMEM reads: a release at cluster scope
// would first wait until the thread's stores to global memory have arrived there (1.9 us in an epilogue).
__device__ __forceinline__ void mbar_arrive_leader(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// commit of a pair's MMAs: arrives on the barrier at the same offset in both CTAs
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}
// One k-block (KSTEPS MMAs per 128-row sub-block) issued from precomputed descriptor
// templates. A single thread issues every MMA of the CTA, so the instruction count
// between two MMAs is what bounds the tensor pipe's duty cycle: the constant descriptor
// fields are assembled once per kernel, and per MMA only the 14-bit start-address field
// (address >> 4) is added in.
template <bool TF32, bool PAIR>
__device__ __forceinline__ void mma_issue(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
#define B2_MMA(GROUP, KIND)                                                    \
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"               \
               "tcgen05.mma." GROUP "." KIND " [%0], %1, %2, %3, p;\n\t}"      \
               ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory")
  if (PAIR && TF32) B2_MMA("cta_group::2", "kind::tf32");
  else if (PAIR) B2_MMA("cta_group::2", "kind::f16");
  else if (TF32) B2_MMA("cta_group::1", "kind::tf32");
  else B2_MMA("cta_group::1", "kind::f16");
#undef B2_MMA
}
// With X3 (fp32-class mode, tf32 only) the stage also holds the low-order
// twins of both slabs, alo16 / blo16 sixteen-byte units behind the slabs themselves, and every
// k-step issues three MMAs: A*B, A*B_lo and A_lo*B (the tensor core truncates fp32 operands
// to tf32, so A and B stand for their own high parts; A_lo*B_lo, 2^-22 of the product, is dropped).
// The two correction products go to an accumulator of their own, X3_CORR_COLS TMEM columns
// behind the main one, and the epilogue adds the two: the tensor core truncates when it adds
// into an accumulator, a bias that grows with the number of additions, so the main sum should
// see K/8 of them, not 3K/8 (measured at K = 4096: 3.0e-5 relative with one accumulator).
template <int SUB, bool TF32, bool PAIR, bool X3, int KS>
__device__ __forceinline__ void issue_ksteps(uint32_t tmem_d, uint64_t adesc0, uint64_t bdesc0, uint32_t a_step16,
                                             uint32_t b_step16, uint32_t idesc, uint32_t block_n, uint32_t accumulate0,
                                             uint32_t a_sub16, uint32_t alo16, uint32_t blo16) {
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    const uint64_t bdesc = bdesc0 + (uint64_t)(ks * b_step16);
    const uint32_t accumulate = ks == 0 ? accumulate0 : 1u;
#pragma unroll
    for (int i = 0; i < SUB; ++i) {  // the 128-row sub-blocks share the B slab
      const uint64_t adesc = adesc0 + (uint64_t)(i * a_sub16 + ks * a_step16);
      const uint32_t d = tmem_d + (uint32_t)i * block_n;
      mma_issue<TF32, PAIR>(d, adesc, bdesc, idesc, accumulate);
      if (X3) {
        mma_issue<TF32, PAIR>(d + X3_CORR_COLS, adesc, bdesc + (uint64_t)blo16, idesc, accumulate);
        mma_issue<TF32, PAIR>(d + X3_CORR_COLS, adesc + (uint64_t)alo16, bdesc, idesc, 1u);
      }
    }
  }
}
template <int SUB_M, bool TF32, bool PAIR, bool X3>
__device__ __forceinline__ void issue_kblock(uint32_t tmem_d, uint64_t adesc0, uint64_t bdesc0, uint32_t a_step16,
                                             uint32_t b_step16, uint32_t idesc, uint32_t block_n, int sub,
                                             bool first_kblock, int ksteps, uint32_t a_sub16, uint32_t alo16 = 0,
                                             uint32_t blo16 = 0) {
  const uint32_t acc0 = first_kblock ? 0u : 1u;
  if (ksteps == KSTEPS) {
    if (SUB_M == 2 && sub == 2)
      issue_ksteps<2, TF32, PAIR, X3, KSTEPS>(tmem_d, adesc0, bdesc0, a_step16, b_step16, idesc, block_n, acc0, a_sub16,
                                              alo16, blo16);
    else
      issue_ksteps<1, TF32, PAIR, X3, KSTEPS>(tmem_d, adesc0, bdesc0, a_step16, b_step16, idesc, block_n, acc0, a_sub16,
                                              alo16, blo16);
  } else {  // half k-blocks
    if (SUB_M == 2 && sub == 2)
      issue_ksteps<2, TF32, PAIR, X3, KSTEPS / 2>(tmem_d, adesc0, bdesc0, a_step16, b_step16, idesc, block_n, acc0,
                                                  a_sub16, alo16, blo16);
    else
      issue_ksteps<1, TF32, PAIR, X3, KSTEPS / 2>(tmem_d, adesc0, bdesc0, a_step16, b_step16, idesc, block_n, acc0,
                                                  a_sub16, alo16, blo16);
  }
}

// 64-bit shared-memory matrix descriptor (version 1) for a 128-byte-swizzled slab.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (Blackwell)
  d |= (uint64_t)layout << 61;
  return d;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* ptr) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}
// ------------------------------------------------------------------ tensor maps (host)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D tensor map over a row-major matrix: `inner` contiguous elements per row,
// `outer` rows, `ld` elements between rows; box = box_inner x box_outer.
// swizzle: 0 = 128 bytes, 1 = 128 bytes in 32-byte atoms, 2 = 64 bytes
bool make_map(CUtensorMap* map, const void* base, int elem_bytes, long long inner, long long outer, long long ld,
              int box_inner, int box_outer, int swizzle) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * elem_bytes};
  cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = enc(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzle == 1 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                   : swizzle == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// 3-D view of an M/N-contiguous operand: {one 128-byte column of M/N, K rows, columns}, so that one
// box holds block_k rows of several columns in the order the slab wants them. `mn` must be a whole number
// of columns (the innermost extent is always a full column, so nothing would be clipped inside it).
bool make_map_columns(CUtensorMap* map, const void* base, int elem_bytes, long long mn, long long k, long long ld,
                      int block_k, int box_columns, int swizzle) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  const int col = SLAB_BYTES / elem_bytes;
  cuuint64_t dims[3] = {(cuuint64_t)col, (cuuint64_t)k, (cuuint64_t)(mn / col)};
  cuuint64_t strides[2] = {(cuuint64_t)ld * elem_bytes, (cuuint64_t)SLAB_BYTES};
  cuuint32_t box[3] = {(cuuint32_t)col, (cuuint32_t)block_k, (cuuint32_t)box_columns};
  cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return enc(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             swizzle == 1 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace b2
