// Host-side helpers shared by the translation units of libb200moe: error reporting and checks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <type_traits>

#include "../../include/b200moe.h"

namespace b200moe {

// codes written by kernels into the caller's `status` word
enum : int {
  ST_OK = 0,
  ST_WAIT_PRODUCER = 1,   // TMA producer: a shared-memory stage never became free
  ST_WAIT_MMA_FULL = 2,   // MMA issuer: a stage never filled
  ST_WAIT_MMA_TMEM = 3,   // MMA issuer: the accumulator was never drained
  ST_WAIT_EPILOGUE = 4,   // epilogue: the accumulator never completed
  ST_BAD_EXPERT_INDEX = 5,// permute: an expert index outside [0, E)
  ST_SELFTEST_TIMEOUT = 6,// self-test: a wait that nothing completes ran out, as intended
  ST_WAIT_PEER = 7,       // cross-rank barrier: a peer's arrival never showed up within the limit
  ST_EP_CAPACITY = 8      // expert parallel with fixed buffers: a rank would receive more rows than its buffers hold
};

void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
int num_sms();
int gemm_cta_budget();   // CTAs a persistent GEMM may occupy (num_sms() minus the reserved SMs)
int exchange_sm_budget();   // SMs (= fat CTAs) the home-side pull kernel of the expert-parallel exchange may occupy

// Elements between rows of the block's own buffers.  A TMA box whose 128-byte rows start 16 bytes past a 32-byte sector moves at three
// quarters of the rate (8.4 against 11.6 TB/s, all from L2; 32 bytes past a line: 10.9), and stores to such rows leave partial sectors: rows whose
// length is no multiple of 64 bytes are padded to whole lines.  us a training pass, dense / padded: 3001 tokens, 32 experts of 1032 x 680, top-4
// 370 / 350; 8192 tokens, 32 of 2056 x 1416 2426 / 2023, of 2040 x 1400 2237 / 1873; 8192 tokens, 16 of 1064 x 2088, top-2 880 / 783; 16 384
// tokens, 64 of 520 x 264, top-6 776 / 722; 2000 tokens, 8 of 264 x 136, top-2 80 / 77.  (Narrow rows grow most: 72 to 128, 8 to 64.)
inline int64_t row_pitch(int64_t n) { return n % 32 == 0 ? n : (n + 63) / 64 * 64; }
// The same where no backward follows, for rows of n that one product over `cols` output columns reads (x_s, inter).  Two tiles of 256 columns read them
// twice only, which at widths below 448 does not pay for the longer rows.  us a forward, all buffers dense / all padded / by this rule: 2571 tokens, 128
// experts of 360 x 256, top-8 81.7 / 83.2 / 81.6; 20 000 tokens, 16 of 136 x 72, top-4 81.5 / 87.4 / 81.4; 20 000, 64 of 392 x 200, top-6 231 / 240 / 231; 8192,
// 32 of 1032 x 680, top-4 278 / 249 / 247; 8192, 128 of 264 x 520, top-8 227 / 211 / 212.
inline int64_t row_pitch_read(int64_t n, int64_t cols) { return cols > 512 || n >= 448 ? row_pitch(n) : n; }
// ... and for rows that no product reads (gate_up, the experts' results), where only their stores gain: dense / padded 8192 tokens, 32 experts of 1544 x 1032
// 455 / 450, of 2056 x 1416 736 / 732, of 1032 x 680 257.6 / 259.2; 20 000 tokens, 16 of 520 x 512 263 / 264, 64 of 392 x 200 237 / 240 (the results alone).
inline int64_t row_pitch_written(int64_t n) { return n >= 1280 ? row_pitch(n) : n; }

// The entry points of the block's steps with the distance between rows given (elements): of x_s, the experts' results and their gradients
// (ldh), of inter (ldi), of gate_up and its gradient (ld2), of any other source (lds)
int gather_rows(const void* x, const int32_t* row_slot, const int32_t* total_rows, int k, int64_t H, int64_t ldh, int64_t rows_cap, void* x_s,
                b200moe_stream_t stream);
int combine_add(const void* rows, int64_t ldh, const float* w, const int32_t* slot_row, const void* add, int64_t T, int k, int64_t H, void* out,
                b200moe_stream_t stream);
int combine_bwd(const void* grad_out, const void* eo, const float* w, const int32_t* row_slot, const int32_t* total_rows, int k, int64_t H,
                int64_t ldh, int64_t rows_cap, void* grad_eo, float* grad_w, b200moe_stream_t stream);
int glu_fwd_rows(const void* gate_up, int64_t ld2, const int32_t* tile_expert, const int32_t* act_codes, const float* act_params,
                 const int32_t* total_rows, int64_t rows_cap, int64_t I, void* inter, int64_t ldi, b200moe_stream_t stream);
int glu_bwd_rows(const void* grad_inter, int64_t ldi, const void* gate_up, int64_t ld2, const int32_t* tile_expert, const int32_t* act_codes,
                 const float* act_params, const int32_t* total_rows, int64_t rows_cap, int64_t I, void* grad_gate_up, float* row_da, float* row_dg,
                 b200moe_stream_t stream);
int special_rows(const void* src, int64_t lds, const int32_t* tile_expert, const int32_t* act_codes, const int32_t* poffs, int first_special,
                 int num_experts, int64_t H, int64_t ldh, int64_t rows_cap, void* dst, b200moe_stream_t stream);
int expert_gate_up(const void* x_s, int64_t ldh, const void* gate_up_proj, const int32_t* act_codes, const int32_t* tile_expert,
                   const int32_t* poffs, int64_t rows_cap, int64_t row_lo, int64_t row_hi, int E, int64_t H, int64_t I, void* gate_up, int64_t ld2,
                   void* inter, int64_t ldi, int32_t* status, b200moe_stream_t stream);
int expert_down_dgrad(const void* grad_eo, int64_t ldh, const void* down_proj, const void* gate_up, int64_t ld2, const int32_t* act_codes,
                      const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int64_t row_lo, int64_t row_hi, int E,
                      int64_t H, int64_t I, void* grad_gate_up, int32_t* status, b200moe_stream_t stream);
int expert_linear(const void* a, int64_t lda, const void* w, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t N,
                  int64_t K, void* out, int64_t ldo, int32_t* status, b200moe_stream_t stream);
int expert_wgrad(const void* A, int64_t lda, const void* B, int64_t ldb, const int32_t* poffs, const int32_t* counts, int64_t rows_cap, int E,
                 int64_t Na, int64_t Nb, void* out, int32_t* status, b200moe_stream_t stream);

// b200moe_permute_build; also stores the counts a second time (counts_out) and adds them to `load` (both nullable)
int permute_build(const int64_t* idx, int64_t T, int k, int E, int32_t* counts, int32_t* offs, int32_t* poffs,
                  int32_t* slot_row, int32_t* row_slot, int32_t* tile_expert, int32_t* order, int32_t* slot_pos, void* ws,
                  size_t ws_bytes, int32_t* counts_out, int64_t* load, int32_t* status, b200moe_stream_t stream);

// router.cu.  counts (nullable): cleared by conv_weight_rows; counts_cleared: some kernel before has done so
int conv_weight_rows(const void* w, int E, int64_t H, int taps, int by_expert, void* wt, int32_t* counts, b200moe_stream_t stream);
int router_topk_fwd(const void* input, int input_kind, const float* bias, int64_t T, int E, int k, int norm_topk, float scale, int64_t* idx,
                    float* w, int32_t* counts, bool counts_cleared, b200moe_stream_t stream);

// gemm_few.cu: whether a forward that no backward follows runs M routed rows over compact rows or over row tiles
bool few_rows_forward(int64_t M, int E, int64_t H, int64_t I);
// its products; early: counts and weights were complete when the kernel in front had passed its wait (FewParams::early)
int expert_gate_up_few(const void* x, const void* gate_up_proj, const int32_t* act_codes, const int32_t* counts,
                       const int32_t* offs, int64_t rows_cap, int E, int64_t H, int64_t I, int early, void* inter,
                       int32_t* status, b200moe_stream_t stream);
int expert_linear_few(const void* x, const void* w, const int32_t* counts, const int32_t* offs, int64_t rows_cap, int E,
                      int64_t N, int64_t K, int early, void* out, int32_t* status, b200moe_stream_t stream);

// gemm.cu: the products of the optimizer's iteration over part of their padded extents
int expert_gram(const void* x, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t K, int mirror,
                int64_t n_live, void* out, int32_t* status, b200moe_stream_t stream);
int expert_linear_axpby(const void* a, const void* w, const void* c, float alpha, float beta, float diag, int symmetric,
                        const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t N, int64_t K,
                        int64_t n_live, int64_t k_live, void* out, int32_t* status, b200moe_stream_t stream);
int expert_linear_t(const void* a, int64_t lda, const void* w, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E,
                    int64_t K, int64_t N, int64_t k_live, void* out, int64_t ldo, int32_t* status, b200moe_stream_t stream);

// Tells the observer set by b200moe_set_observer, if any, where an operation of a longer sequence begins and ends
struct OpScope {
  OpScope(const char* name, int launches);
  ~OpScope();
  const char* name;
  int launches;
};

#define B200_CHECK_ARG(cond, code, ...)  \
  do {                                   \
    if (!(cond)) {                       \
      ::b200moe::set_error(__VA_ARGS__); \
      return (code);                     \
    }                                    \
  } while (0)

#define B200_CUDA(call)                                                   \
  do {                                                                    \
    cudaError_t e__ = (call);                                             \
    if (e__ != cudaSuccess) return ::b200moe::cuda_fail(e__, #call);      \
  } while (0)

// f(TPR): threads of a 256-thread CTA that share a row of nvec 16-byte vectors in the copying kernels, at least 32
template <class F>
inline void by_row_threads(int nvec, F f) {
  if (nvec <= 32) f(std::integral_constant<int, 32>());
  else if (nvec <= 64) f(std::integral_constant<int, 64>());
  else if (nvec <= 128) f(std::integral_constant<int, 128>());
  else f(std::integral_constant<int, 256>());
}

// Launch whose set-up may overlap the end of the kernel before it in the stream (programmatic stream serialisation).  Every
// kernel launched this way calls grid_dep_wait() (ptx.cuh) in all of its threads before it reads or writes anything that
// another kernel touches, and grid_dep_launch() only after that: when a kernel's first instruction runs, the kernel two
// before it is complete, and past its wait the one before it too.  What those wrote is visible past the wait only: nothing orders a
// kernel's first reads behind writes that another kernel waited for.  (Products of a backward that neither wait for the one before them nor need
// anything of it took 3 % off a pass of 3001 tokens, 32 experts of 1032 x 680; nothing that the programming model states made them correct.)  One
// exception, FewParams::early in gemm_few.cu, says there what it rests on.
// A kernel's pointers are neither __restrict__ nor read by __ldg: both
// promise the compiler data that stays as it is for the kernel's whole life, which begins before the wait, so it could load ahead
// of the wait or past the coherent cache.  (Taking the promises out cost next to nothing: combine of 98 304 rows of 2048 96.4 /
// 96.3 us, both quantisers of them 186 / 184, GLU backward of 1408 columns 457 / 457, the conv router's pass 115.0 / 115.3.)  Why: between two plain launches the SMs idle for 1.5 to 4
// us (drain, launch, barriers, tensor memory, descriptors), as long as the small kernels of a decoding step run.  The GEMMs
// call grid_dep_launch() when their last loads are issued: early enough to hide a launch, and at their start it made large
// training steps 1 % slower.  us a pass, plain / chained: 48 tokens, 64 experts of 2048 x 1408 (6 launches, with the weights
// ahead of the wait, gemm_few.cu) 205 / 192; 1500 tokens 297 / 285; forward and backward of 3001 tokens, 32 experts of 1032 x
// 680 (18 launches) 415 / 381; mixed stack of 16 384 tokens 408 / 384.
// With SMs reserved for an exchange (b200moe_set_reserved_sms) the launch is a plain one: CTAs that wait would sit on them.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (gemm_cta_budget() == num_sms()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#define B200_LAUNCH(kernel, grid, block, smem, stream, ...) \
  B200_CUDA(::b200moe::launch_chained(kernel, grid, block, smem, (cudaStream_t)(stream), 1, __VA_ARGS__))

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace b200moe
