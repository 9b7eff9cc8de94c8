// Shared declarations of the b200mlp CUDA sources (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace b2 {

enum Epilogue : int {
  EPI_NONE = 0,  // C = alpha * acc (+ beta * C)
  EPI_RELU = 1,  // C = max(acc, 0)                    forward of a hidden layer
  EPI_MASK = 2   // C = aux > 0 ? acc : 0              input gradient through a ReLU
};

enum ElemType : int { T_F32 = 0, T_BF16 = 1 };

// One GEMM, C[M x N] = op(A) * op(B), described by element strides so that the
// three call forms of the training step share every kernel:
//   forward  (NoTrans x Trans)   A(m,k) = A[m*lda + k]   B(k,n) = B[n*ldb + k]
//   wgrad    (Trans   x NoTrans) A(m,k) = A[k*lda + m]   B(k,n) = B[k*ldb + n]
//   dgrad    (NoTrans x NoTrans) A(m,k) = A[m*lda + k]   B(k,n) = B[k*ldb + n]
struct GemmDesc {
  int M, N, K;
  const void* A;
  long long sAm, sAk;
  const void* B;
  long long sBk, sBn;
  void* C;
  long long ldc;
  const void* aux;  // EPI_MASK only, same element type as A/B operands
  long long ldaux;
  float alpha, beta;
  int epilogue;
  int in_type;   // ElemType of A, B and aux
  int out_type;  // ElemType of C
  int pad_writable;  // 1: the bytes between column N and the next 16-byte boundary of a row of C may be overwritten
  int shared_sms;    // 1: another library's kernels may hold some of the SMs while this GEMM runs
  int large_tiles;   // 1: CUDA-core GEMM: not the kernel for small grids
  // Optional stream-K workspace of the tensor-core kernel (null = whole tiles per CTA):
  // TC_WS_SLOT_BYTES per SM and one zero-initialised flag word per SM. GEMMs that share a
  // workspace must not overlap on the GPU.
  float* ws;
  unsigned int* ws_flags;
  // fp32-class tensor-core mode (in_type T_F32 only): low-order twins x - tf32(x) of both
  // operands (same shapes and strides as A and B). With both set the kernel issues three tf32
  // MMAs per k-step (A*B + A*B_lo + A_lo*B), which restores fp32-class accuracy. C_lo (same
  // shape and ldc as C, fp32) receives the twin of the result for the GEMM that reads C next.
  const void* A_lo;
  const void* B_lo;
  void* C_lo;
  // Optional in-kernel timeline of the tensor-core kernel (null = off): CTA 0 stamps %globaltimer
  // per tile into trace[tile * 4 + {0: first MMA issued, 1: accumulator complete (seen by the
  // epilogue), 2: accumulator released, 3: last store of the tile issued}], up to TC_TRACE_TILES tiles.
  // Behind them, for the first TC_TRACE_KBLOCKS k-blocks of CTA 0's second tile: when the MMA warp
  // saw the k-block's operands in shared memory, when the TMA warp saw the k-block's slot free, and
  // (CTA-pair kernel) when the peer CTA's TMA warp saw it free.
  unsigned long long* trace;
};
constexpr int TC_TRACE_TILES = 64;
constexpr int TC_TRACE_KBLOCKS = 64;
constexpr int TC_TRACE_WORDS = TC_TRACE_TILES * 4 + 3 * TC_TRACE_KBLOCKS;
constexpr size_t TC_WS_SLOT_BYTES = 2 * 128 * 256 * sizeof(float);

// CUDA-core GEMM for any shape, stride and alignment (fp32 accumulate).
cudaError_t gemm_simt_launch(const GemmDesc& g, cudaStream_t stream);
// Kernel for small grids (gemm_f32.cu), which gemm_simt_launch takes where it serves and large_tiles is not set.
bool gemm_f32_serves(const GemmDesc& g);
cudaError_t gemm_f32_launch(const GemmDesc& g, cudaStream_t stream);
bool gemm_simt_small(const GemmDesc& g);  // served by one of its kernels for small grids (unless large_tiles)
double gemm_simt_us(const GemmDesc& g);  // estimate (fp32)
bool gemm_simt_short_sums(const GemmDesc& g);  // its sums are partial ones of K / 16 or K / 32 terms and not one in k order

// GEMM of fp32 matrices on the tensor cores at fp32 precision, any alignment (gemm_split.cu), where it is faster than
// gemm_simt_launch; on at most `sms` SMs, which decide that too; `status` as for gemm_tc_launch.
bool gemm_split_serves(const GemmDesc& g, int sms);
double gemm_split_us(const GemmDesc& g, int sms);  // estimate
cudaError_t gemm_split_launch(const GemmDesc& g, int sms, cudaStream_t stream, unsigned int* status);

// Tensor-core (tcgen05 + TMA + TMEM) GEMM. in_type T_BF16 -> kind::f16 (bf16),
// in_type T_F32 -> kind::tf32. Returns cudaErrorNotSupported when the shape or
// alignment cannot be served (caller falls back to gemm_simt_launch).
// `status` is a device word the kernel sets non-zero if a bounded wait gave up.
struct TcPlan;  // opaque: tensor maps + tile choice for one GEMM site
TcPlan* gemm_tc_plan_create(const GemmDesc& g, int sm_count, char* err, size_t errlen);
void gemm_tc_plan_destroy(TcPlan* p);
// ReLU bit plane of a plan (one bit per element of C, words of 32 columns, ld_words words per
// row): mask_out on a forward plan with the ReLU epilogue, mask_in on an input-gradient plan with
// the mask epilogue (read instead of the activation). False when the plan cannot use one.
bool gemm_tc_plan_set_mask(TcPlan* plan, uint32_t* mask_out, const uint32_t* mask_in, long long ld_words);
cudaError_t gemm_tc_launch(const TcPlan* p, cudaStream_t stream, unsigned int* status);

// Whole training steps as one launch (step_kernel.cu). The GEMMs of a step in an order in which each depends
// only on earlier ones, with what its tiles wait for (indices into `gemms`, -1: nothing).
enum StepRole : int { STEP_GEMM = 0, STEP_LAST_FWD = 1, STEP_WGRAD = 2 };
struct StepGemm {
  GemmDesc d;
  int role;          // STEP_LAST_FWD: the epilogue also writes dz and the loss; STEP_WGRAD: it also updates w
  int block_n;       // tile width, 64 or 128 (128 for pairs)
  int rows_of;       // a tile needs the same row block of that GEMM's result
  int all_of;        // a tile needs that GEMM's whole result
  int update_after;  // STEP_WGRAD: w may change once that GEMM (which reads it) is done
  int mask_of;       // the GEMM that writes mask_in
  int prev_step[2];  // weight gradients of the previous step that must be done, update included
  uint32_t* mask_out;
  const uint32_t* mask_in;
  long long ld_mask;
  float* w;
  __nv_bfloat16* w16;
  float* w_lo;
};
struct StepSpec {
  std::vector<StepGemm> gemms;
  bool pair;  // tiles of 256 x 128 by CTA pairs
  const float* target;
  void* dz;
  float* dz_lo;
  int baseline;
  float inv_batch;
  double loss_scale;
  double* loss;
};
struct StepPlan;
int step_plan_counters(const StepSpec& s);  // counter words a launch needs, zeroed by the caller before it
StepPlan* step_plan_create(const StepSpec& s, int sm_count);  // null: cannot be served
void step_plan_destroy(StepPlan* p);
cudaError_t step_launch(const StepPlan* plan, int steps, float lr, unsigned int* counters, unsigned int* status,
                        cudaStream_t stream);

constexpr unsigned int STATUS_GRID_BARRIER = 16;  // the status word where a wait of small_step.cu gave up
// Whole steps of small fp32 networks as one cooperative launch (small_step.cu). Rows of all matrices are dense.
constexpr int SMALL_LAYERS = 16;
enum SmallForm : int { SMALL_FWD = 0, SMALL_DGRAD = 1, SMALL_WGRAD = 2 };
struct SmallLayer {
  int fi, fo;
  bool short_sums[3];  // by form: gemm_simt_short_sums of the GEMM
  const float* in;  // batch x fi
  float* out;       // batch x fo: the next layer's input, or the network's output
  float* dz;        // batch x fo
  float* dx;        // batch x fi: the layer's below dz, or the input gradient
  float *w, *dw;    // fo x fi
};
struct SmallStep {
  SmallLayer layer[SMALL_LAYERS];
  int L, batch, baseline, input_grad;
  const float* target;
  float inv_batch;
  double loss_scale;
  double* loss;
};
bool small_step_serves(const SmallStep& s, int sms, double launches_us);  // launches_us: a step as a launch per GEMM
int small_step_steps(const SmallStep& s, int sms);  // that one launch should take
int small_step_blocks(const SmallStep& s, int sms);
// Barriers of a launch: each adds `blocks` to *counter, which stands at `count` before the launch. A launch that finds *status
// set (a wait of an earlier one gave up, so the counter is behind) touches neither counter nor weights.
int small_step_barriers(const SmallStep& s, int steps);
cudaError_t small_step_launch(const SmallStep& s, int blocks, int steps, float lr, unsigned int count, unsigned int* counter,
                              unsigned int* status, cudaStream_t stream);

// Small-message allreduce over peer memory (p2p_allreduce.cu). Every rank's gradient slab and
// flag block are addressable from every rank (peer access within a process, IPC mappings
// between processes). A flag block is 2 * P2P_MAX_RANKS words, written by the peers: word
// P2P_FLAG_ARRIVE + r = "rank r's input of call `epoch` is ready", P2P_FLAG_DONE + r = "rank r's
// stores of call `epoch` are done".
constexpr int P2P_MAX_RANKS = 8;
constexpr int P2P_FLAG_ARRIVE = 0;
constexpr int P2P_FLAG_DONE = P2P_MAX_RANKS;
constexpr size_t P2P_FLAG_BYTES = 2 * P2P_MAX_RANKS * sizeof(unsigned int);
struct P2pParams {
  float* slab[P2P_MAX_RANKS];          // index = rank; slab[rank] is this rank's own
  unsigned int* flags[P2P_MAX_RANKS];  // index = rank
  int world, rank;
  unsigned long long offset;  // first element of the message in every slab (multiple of 4)
  unsigned long long count;   // elements
  unsigned int epoch;         // call counter, > 0, the same on every rank for the same call
  unsigned int* ctas_done;    // this rank's own counter, zero between calls
  unsigned int* status;       // this rank's own word, set non-zero when a wait gave up
  unsigned long long wait_ns; // how long a flag wait may last before the rank gives up
};
// One rank's launch (every rank launches its own, each on its own GPU).
cudaError_t p2p_allreduce_launch(const P2pParams& p, int cta_limit, cudaStream_t stream);
// All ranks in one cooperative launch on one GPU: `ranks_dev` = device array of world entries.
cudaError_t p2p_allreduce_emulated_launch(const P2pParams* ranks_dev, const P2pParams& any_rank, cudaStream_t stream);

// Element-wise kernels.
// For the current device: the kernels that prepare the next host-fed batch ask for the shared-memory split the GEMM
// kernels run with, so that an SM need not drain before it takes them beside a running step. (The weight update
// is not among them: with it 8 x 4096 layers, 1024 rows, bf16 took 1042 us per step against 1032.)
cudaError_t elementwise_prepare();
cudaError_t convert_f32_to_bf16(const float* src, __nv_bfloat16* dst, size_t n, cudaStream_t s);
cudaError_t convert_bf16_to_f32(const __nv_bfloat16* src, float* dst, size_t n, cudaStream_t s);
// dz = y (ref) or (y - t) * inv_batch (baseline); loss += 0.5 * sum(d^2) * loss_scale. Rows of `pitch` elements (a
// multiple of 4 where it is not `cols`); dz is zero behind column cols.
cudaError_t loss_grad_launch(const float* y, const float* target, void* dz, int dz_type, int rows, int cols,
                             int pitch, int baseline, float inv_batch, double loss_scale, double* loss,
                             cudaStream_t s, float* dz_lo = nullptr);
// w = fma(-lr, g, w); optional bf16 copy of the new weights, optional low-order twin w - tf32(w)
cudaError_t sgd_launch(float* w, const void* g, int g_type, __nv_bfloat16* w_bf16, size_t n, float lr,
                       int sm_count, cudaStream_t s, float* w_lo = nullptr);
// *out += sum of the 32-bit words of buf modulo 2^64 (out must be zeroed by the caller)
cudaError_t fingerprint_launch(const void* buf, size_t bytes, unsigned long long* out, cudaStream_t s);
// The same for rows x cols 16-bit elements stored with a row pitch of ld elements, paired into words as if
// the rows were dense (a last unpaired element is left out, as by fingerprint_launch)
cudaError_t fingerprint_rows16_launch(const void* buf, int rows, int cols, int ld, unsigned long long* out,
                                      cudaStream_t s);
// dst = src - tf32(src): the part of an fp32 value the tensor core drops when it reads it as tf32
cudaError_t split_lo_launch(const float* src, float* dst, size_t n, cudaStream_t s);
cudaError_t fill_uniform_launch(void* buf, int type, size_t n, uint64_t seed, float lo, float hi,
                                cudaStream_t s);

}  // namespace b2
