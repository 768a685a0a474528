// The whole block from one host call: router, permutation, expert GEMMs, activation, combine, forward and backward, as
// one sequence of the library's own launches on the caller's stream, out of one workspace that the caller
// allocates (the *_ws_bytes functions give its size, `carve_*` its layout).  Nothing here touches the device but the
// launches; the forward's workspace is what a backward reads, so it must stay as the forward left it until then.
//
// Why: a launch from here costs the host about 2 us; through one Python call, its output allocations and argument
// checks per kernel it cost 8 to 15 us, more than most kernels of a small batch run on the GPU.
// A pass among others: one decoding token 165 -> 65 us (10 -> 6 launches), forward and backward of 512 tokens at width 256
// 607 -> 266 us (24 -> 17), ragged training step (3001 tokens, H 1032, I 680, 32 experts) 625 -> 515 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace b200moe {

typedef uint16_t bf16_t;   // storage only

struct Carver {
  char* base;
  size_t off;
  explicit Carver(void* p) : base(static_cast<char*>(p)), off(0) {}
  template <class T>
  T* take(int64_t n) {
    off = (off + 255) & ~static_cast<size_t>(255);
    T* p = base != nullptr ? reinterpret_cast<T*>(base + off) : nullptr;
    off += static_cast<size_t>(n) * sizeof(T);
    return p;
  }
};

enum Kind { KIND_FEW = 0, KIND_TILES = 1, KIND_ROWS = 2 };

struct Dims {
  int64_t T, H, I;
  int E, n_glu, k;        // routed experts, those with weights, picks per token
  int keep;               // whether a backward may follow
  Kind kind;
  int64_t M() const { return T * k; }
  int64_t rows() const { return kind == KIND_FEW ? M() : b200moe_padded_rows_cap(M(), E); }
  // elements between rows of x_s, of the experts' results and their gradient, of inter, of gate_up (row_pitch; the few-rows kernels take dense ones).
  // Where no backward follows, a product reads x_s and inter only.
  int64_t ldx() const { return keep ? row_pitch(H) : kind == KIND_FEW ? H : row_pitch_read(H, 2 * I); }
  int64_t ldh() const { return keep ? row_pitch(H) : kind == KIND_FEW ? H : row_pitch_written(H); }
  int64_t ldi() const { return keep ? row_pitch(I) : kind == KIND_FEW ? I : row_pitch_read(I, H); }
  int64_t ld2() const { return keep ? row_pitch(2 * I) : row_pitch_written(2 * I); }
};

static Dims make_dims(int64_t T, int64_t H, int64_t I, int E, int n_glu, int k, int keep, int rows_kernels) {
  Dims d{T, H, I, E, n_glu, k, keep, KIND_TILES};
  if (rows_kernels) d.kind = KIND_ROWS;
  else if (!keep && T > 0 && k > 0 && E > 0 && few_rows_forward(T * k, E, H, I)) d.kind = KIND_FEW;
  return d;
}

static int check_dims(const char* who, const Dims& d) {
  B200_CHECK_ARG(d.T > 0 && d.H > 0 && d.I > 0 && d.H % 8 == 0 && d.I % 8 == 0 && d.E >= 1 && d.n_glu >= 1 && d.n_glu <= d.E &&
                     d.k >= 1 && d.T < (1LL << 31),
                 B200MOE_E_BAD_SHAPE, "%s: T = %lld, H = %lld, I = %lld (multiples of 8), E = %d (%d with weights), k = %d", who,
                 (long long)d.T, (long long)d.H, (long long)d.I, d.E, d.n_glu, d.k);
  return 0;
}

struct Forward {
  int32_t *counts, *offs, *poffs, *slot_row, *row_slot, *tile_expert, *order, *slot_pos;
  void* scratch;
  size_t scratch_bytes;
  bf16_t *x_s, *gate_up, *inter, *eo;
  bf16_t* logits;         // of the router, when it runs here
  int64_t* idx;
  float* w;
};

static Forward carve_forward(const Dims& d, bool router, void* ws, size_t* bytes) {
  Carver c(ws);
  Forward f{};
  const int64_t M = d.M(), cap = b200moe_padded_rows_cap(M, d.E), rows = d.rows();
  const bool few = d.kind == KIND_FEW;
  f.counts = c.take<int32_t>(d.E);
  f.offs = c.take<int32_t>(d.E + 1);
  f.poffs = c.take<int32_t>(d.E + 1);
  f.slot_row = c.take<int32_t>(M);
  f.row_slot = c.take<int32_t>(cap);
  f.tile_expert = c.take<int32_t>(cap / B200MOE_TILE_M);
  if (few) {
    f.order = c.take<int32_t>(M);
    f.slot_pos = c.take<int32_t>(M);
  }
  f.scratch_bytes = b200moe_permute_ws_bytes(M, d.E);
  f.scratch = c.take<char>(f.scratch_bytes);
  if (router) {
    f.logits = c.take<bf16_t>(d.T * d.E);
    f.idx = c.take<int64_t>(M);
    f.w = c.take<float>(M);
  }
  f.x_s = c.take<bf16_t>(rows * d.ldx());
  if (!few) f.gate_up = c.take<bf16_t>(rows * d.ld2());
  f.inter = c.take<bf16_t>(rows * d.ldi());
  f.eo = c.take<bf16_t>(rows * d.ldh());
  if (bytes != nullptr) *bytes = c.off;
  return f;
}

struct Backward {
  bf16_t *grad_eo, *grad_gu, *grad_x_s, *grad_inter;
  float *row_da, *row_dg;
  float* grad_w;                     // when the router's backward follows
  bf16_t *grad_logits, *grad_x_router;
  float* part;
};

// Split-K of the router's weight gradient dW (E, H) = gl (T, E)^T x (T, H).  Up to 128 experts the product runs as
// dW^T = x^T gl, whose rows (H) fill the MMA's M; gl^T x would multiply E of 256 rows.  About one tile per SM; the slices
// are summed, and transposed back, by the reduction.  T 16384, H 2048, 64 experts: product + reduction 48 -> 31 us.
//
// `sms`: the SMs the GEMM may use.  A launch takes gemm_cta_budget(), which shrinks while SMs are reserved for an exchange;
// a workspace is sized for num_sms(), which never gives fewer slices.
struct Split { int64_t chunk, slices; };
static Split split_k(int64_t T, int64_t tiles, int64_t per_wave) {
  if (T <= 0) return {64, 0};
  const int64_t want = std::max<int64_t>(1, std::min<int64_t>(per_wave / std::max<int64_t>(tiles, 1), (T + 63) / 64));
  const int64_t chunk = ((T + want - 1) / want + 63) / 64 * 64;
  return {chunk, (T + chunk - 1) / chunk};
}
static bool router_dw_transposed(int64_t E) { return E <= 128; }
static Split router_split(int64_t T, int64_t E, int64_t H, int sms) {
  if (router_dw_transposed(E)) return split_k(T, ((H + 127) / 128) * ((E + 127) / 128), sms);
  return split_k(T, ((E + 127) / 128) * ((H + 255) / 256), 2 * sms);
}

static Backward carve_backward(const Dims& d, bool router, void* ws, size_t* bytes) {
  Carver c(ws);
  Backward b{};
  const int64_t rows = d.rows();
  b.grad_eo = c.take<bf16_t>(rows * d.ldh());
  b.grad_gu = c.take<bf16_t>(rows * d.ld2());
  if (d.kind == KIND_ROWS) {
    b.grad_x_s = c.take<bf16_t>(rows * d.ldh());       // grad_eo is still read (Identity experts) while this is written
    b.grad_inter = c.take<bf16_t>(rows * d.ldi());
    b.row_da = c.take<float>(rows);
    b.row_dg = c.take<float>(rows);
  } else {
    b.grad_x_s = b.grad_eo;                        // written after the last read of grad_eo
  }
  if (router) {
    b.grad_w = c.take<float>(d.M());
    b.grad_logits = c.take<bf16_t>(d.T * d.E);
    b.grad_x_router = c.take<bf16_t>(d.T * d.H);
    b.part = c.take<float>(router_split(d.T, d.E, d.H, num_sms()).slices * d.E * d.H);
  }
  if (bytes != nullptr) *bytes = c.off;
  return b;
}

#define RUN(name, launches, call)     \
  do {                                \
    OpScope scope__(name, launches);  \
    const int rc__ = (call);          \
    if (rc__) return rc__;            \
  } while (0)

static int permute(const Dims& d, const int64_t* idx, const Forward& f, int32_t* counts_out, int64_t* load, int32_t* status,
                   b200moe_stream_t st) {
  RUN("permute_build", d.M() > 1024 ? 2 : 1,
      permute_build(idx, d.T, d.k, d.E, f.counts, f.offs, f.poffs, f.slot_row, f.row_slot, f.tile_expert, f.order,
                    f.slot_pos, f.scratch, f.scratch_bytes, counts_out, load, status, st));
  return 0;
}

static int experts_forward(const Dims& d, const void* x, const float* w, const void* gate_up_proj, const void* down_proj,
                           const int32_t* codes, const float* params, const Forward& f, void* out, int32_t* status,
                           b200moe_stream_t st) {
  const int64_t rows = d.rows();
  if (d.kind == KIND_FEW) {
    RUN("gather_rows", 1, b200moe_gather_rows(x, f.order, f.offs + d.E, d.k, d.H, rows, f.x_s, st));
    // early: past its wait the gather has the permutation behind it, and the permutation whatever wrote the weights
    RUN("expert_gate_up_few", 1, expert_gate_up_few(f.x_s, gate_up_proj, codes, f.counts, f.offs, rows, d.E, d.H, d.I, 1, f.inter,
                                                    status, st));
    RUN("expert_linear_few", 1, expert_linear_few(f.inter, down_proj, f.counts, f.offs, rows, d.E, d.H, d.I, 1, f.eo, status, st));
    RUN("combine", 1, b200moe_combine(f.eo, w, f.slot_pos, d.T, d.k, d.H, out, st));
    return 0;
  }
  const int64_t ldx = d.ldx(), ldh = d.ldh(), ldi = d.ldi(), ld2 = d.ld2();
  RUN("gather_rows", 1, gather_rows(x, f.row_slot, f.poffs + d.E, d.k, d.H, ldx, rows, f.x_s, st));
  if (d.kind == KIND_TILES) {
    RUN("expert_gate_up_swiglu", 1, expert_gate_up(f.x_s, ldx, gate_up_proj, codes, f.tile_expert, f.poffs, rows, 0, 0, d.E, d.H, d.I,
                                                   f.gate_up, ld2, f.inter, ldi, status, st));
    RUN("expert_down", 1, expert_linear(f.inter, ldi, down_proj, f.tile_expert, f.poffs, rows, d.E, d.H, d.I, f.eo, ldh, status, st));
  } else {   // the GEMMs and the activation kernels see the rows of the experts with weights only
    RUN("expert_linear", 1, expert_linear(f.x_s, ldx, gate_up_proj, f.tile_expert, f.poffs, rows, d.n_glu, 2 * d.I, d.H, f.gate_up, ld2, status, st));
    RUN("glu_fwd_rows", 1, glu_fwd_rows(f.gate_up, ld2, f.tile_expert, codes, params, f.poffs + d.n_glu, rows, d.I, f.inter, ldi, st));
    RUN("expert_linear", 1, expert_linear(f.inter, ldi, down_proj, f.tile_expert, f.poffs, rows, d.n_glu, d.H, d.I, f.eo, ldh, status, st));
    if (d.n_glu < d.E)
      RUN("special_rows", 1, special_rows(f.x_s, ldx, f.tile_expert, codes, f.poffs, d.n_glu, d.E, d.H, ldh, rows, f.eo, st));
  }
  RUN("combine", 1, combine_add(f.eo, ldh, w, f.slot_row, nullptr, d.T, d.k, d.H, out, st));
  return 0;
}

// Gradients to compute (nullptr: not wanted; x != nullptr: the rows b.grad_x_s, which the caller combines per token)
struct Grads {
  void *x, *gate_up, *down;
  float *w, *params;
};

static int experts_backward(const Dims& d, const void* grad_out, const float* w, const void* gate_up_proj,
                            const void* down_proj, const int32_t* codes, const float* params, const Forward& f,
                            const Backward& b, const Grads& g, int32_t* status, b200moe_stream_t st) {
  const int64_t rows = d.rows();
  const int32_t* total = f.poffs + d.E;
  const int64_t ldh = d.ldh(), ldi = d.ldi(), ld2 = d.ld2();
  RUN("combine_bwd", 1, combine_bwd(grad_out, f.eo, w, f.row_slot, total, d.k, d.H, ldh, rows, b.grad_eo, g.w, st));
  const int n = d.n_glu;
  float* da = g.params != nullptr ? b.row_da : nullptr;
  float* dg = g.params != nullptr ? b.row_dg : nullptr;
  if (d.kind == KIND_ROWS) {
    RUN("expert_linear_t", 1, expert_linear_t(b.grad_eo, ldh, down_proj, f.tile_expert, f.poffs, rows, n, d.H, d.I, d.H, b.grad_inter, ldi, status, st));
    RUN("glu_bwd_rows", 1, glu_bwd_rows(b.grad_inter, ldi, f.gate_up, ld2, f.tile_expert, codes, params, f.poffs + n, rows, d.I, b.grad_gu, da, dg, st));
  } else if (g.x != nullptr || g.gate_up != nullptr) {
    RUN("expert_down_dgrad_glu", 1, expert_down_dgrad(b.grad_eo, ldh, down_proj, f.gate_up, ld2, codes, f.tile_expert, f.poffs, rows, 0, 0,
                                                      d.E, d.H, d.I, b.grad_gu, status, st));
  }
  if (g.down != nullptr)
    RUN("expert_wgrad", 1, expert_wgrad(b.grad_eo, ldh, f.inter, ldi, f.poffs, f.counts, rows, n, d.H, d.I, g.down, status, st));
  if (g.gate_up != nullptr)
    RUN("expert_wgrad", 1, expert_wgrad(b.grad_gu, ld2, f.x_s, ldh, f.poffs, f.counts, rows, n, 2 * d.I, d.H, g.gate_up, status, st));
  if (g.x != nullptr) {
    RUN(d.kind == KIND_ROWS ? "expert_linear_t" : "expert_gate_up_dgrad", 1,
        expert_linear_t(b.grad_gu, ld2, gate_up_proj, f.tile_expert, f.poffs, rows, n, 2 * d.I, d.H, 2 * d.I, b.grad_x_s, ldh, status, st));
    if (d.kind == KIND_ROWS && n < d.E)
      RUN("special_rows", 1, special_rows(b.grad_eo, ldh, f.tile_expert, codes, f.poffs, n, d.E, d.H, ldh, rows, b.grad_x_s, st));
  }
  if (g.params != nullptr) {
    if (n < d.E)
      B200_CUDA(cudaMemsetAsync(g.params + 2 * n, 0, sizeof(float) * 2 * (d.E - n), (cudaStream_t)st));
    RUN("expert_row_sums", 1, b200moe_expert_row_sums(da, dg, f.poffs, n, g.params, st));
  }
  return 0;
}

// Up to 16 tokens per SM and 128 experts logits and picks are one launch (gemm_few.cu, with the times of both)
constexpr int64_t kSmallTokensPerSm = 16;
constexpr int kSmallExperts = 128;

static int router_forward(const void* x, const void* weight, const float* bias, int64_t T, int64_t H, int E, int k, int norm,
                          float scale, void* logits, int64_t* idx, float* w, int32_t* counts, int32_t* status,
                          b200moe_stream_t st) {
  if (T <= kSmallTokensPerSm * num_sms() && E <= kSmallExperts) {
    RUN("router_small_fwd", 1, b200moe_router_small_fwd(x, weight, bias, T, H, E, k, norm, scale, logits, idx, w, counts, status, st));
    return 0;
  }
  RUN("gemm_nt", 1, b200moe_gemm_nt(x, weight, logits, T, E, H, status, st));
  RUN("router_topk_fwd", 1, b200moe_router_topk_fwd(logits, B200MOE_LOGITS_BF16, bias, T, E, k, norm, scale, idx, w, counts, st));
  return 0;
}

static int router_backward(const void* x, const void* weight, const void* logits, const int64_t* idx, const float* grad_w,
                           int64_t T, int64_t H, int E, int k, int norm, float scale, void* grad_logits, float* part,
                           void* grad_x, void* grad_weight, int32_t* status, b200moe_stream_t st) {
  RUN("router_topk_bwd", 1, b200moe_router_topk_bwd(logits, B200MOE_LOGITS_BF16, idx, grad_w, T, E, k, norm, scale, grad_logits, st));
  if (grad_x != nullptr) RUN("gemm_nn", 1, b200moe_gemm_nn(grad_logits, weight, grad_x, T, H, E, status, st));
  if (grad_weight != nullptr) {
    OpScope scope("gemm_tn", 2);
    const Split sp = router_split(T, E, H, gemm_cta_budget());
    const bool tr = router_dw_transposed(E);
    int rc = tr ? b200moe_gemm_tn_splitk(x, grad_logits, part, H, E, T, sp.chunk, status, st)
                : b200moe_gemm_tn_splitk(grad_logits, x, part, E, H, T, sp.chunk, status, st);
    if (rc) return rc;
    rc = tr ? b200moe_splitk_reduce_t(part, sp.slices, H, E, grad_weight, st)
            : b200moe_splitk_reduce(part, sp.slices, static_cast<int64_t>(E) * H, grad_weight, st);
    if (rc) return rc;
  }
  return 0;
}

// ---- conv router.  logits[s] = sum_j x[s - (taps-1) + j] W_j^T with W_j (E, H): one GEMM over (tap, channel) whose
// producer shifts its boxes of x (gemm.cu).  Backward: the top-k kernel writes u (T, taps*E), every tap's gradient beside the
// row of x it belongs to, and dX = u [W_j], dW = u^T x are plain products that read x and write dX once, for all taps, at
// any sequence length.  x (16, 1024, 2048), 64 experts, 4 taps: dW 69 -> 26 us against a product that shifts x tap by tap
// (E of 256 MMA rows, x read four times).
// (The same turn of the forward, z = x [W_j]^T and adding its rows up, reads x once as well, but adds in another order: 1 in
// 7000 picks of close experts then differs, and a token's gradient with it.)
static Split conv_split(int64_t T, int64_t rows, int64_t H, int sms) {   // one wave of pair tiles, up to 128 rows of single-CTA tiles
  if (rows <= 128) return split_k(T, (H + 127) / 128, sms);
  return split_k(T, ((rows + 255) / 256) * ((H + 255) / 256), sms / 2);
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

// ---------------------------------------------------------------------------- router alone
int b200moe_router_forward(const void* x, const void* weight, const float* bias, int64_t T, int64_t H, int E, int k,
                           int norm_topk, float scale, void* logits, int64_t* idx, float* w, int32_t* counts,
                           int32_t* status, b200moe_stream_t stream) {
  return router_forward(x, weight, bias, T, H, E, k, norm_topk, scale, logits, idx, w, counts, status, stream);
}

size_t b200moe_router_bwd_ws_bytes(int64_t T, int64_t H, int E) {
  if (T <= 0 || H <= 0 || E <= 0) return 0;
  Carver c(nullptr);
  c.take<bf16_t>(T * E);
  c.take<float>(router_split(T, E, H, num_sms()).slices * E * H);
  return c.off;
}

int b200moe_router_backward(const void* x, const void* weight, const void* logits, const int64_t* idx, const float* grad_w,
                            int64_t T, int64_t H, int E, int k, int norm_topk, float scale, void* ws, void* grad_x,
                            void* grad_weight, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(ws, B200MOE_E_NULL, "router_backward: null workspace");
  Carver c(ws);
  bf16_t* gl = c.take<bf16_t>(T * E);
  float* part = c.take<float>(router_split(T, E, H, num_sms()).slices * E * H);
  return router_backward(x, weight, logits, idx, grad_w, T, H, E, k, norm_topk, scale, gl, part, grad_x, grad_weight, status, stream);
}

// ---------------------------------------------------------------------------- conv router
// In place or over an unfolded copy of x (the same k order, so the same logits to the bit).  In place the row tiles lie in one
// sequence each and the k-blocks in one tap each, so short sequences and widths that are no multiple of 64 multiply padding;
// the copy writes taps * H values per token and takes two more launches.  Both run waves of tiles of one accumulator chain:
// compared are the k-blocks of their waves, 0.31 us each, with 22 of them for the launches and one per 1.9 MB of copy.  us, in
// place / unfolded, 64 experts, 4 taps, H 2048, 16 384 tokens in sequences of 1: 4290 / 119, 16: 273 / 120, 48: 124 / 120,
// 64: 85 / 120, 128: 47 / 120; of 4096 tokens in sequences of 16: 85 / 56, 32: 43 / 56; H 80, 16 384 tokens in sequences of 1:
// 326 / 19, 16: 25 / 18, 32: 15 / 18.
// A width that is no multiple of 16 would split an MMA's 16 channels between taps: always unfolded.
static bool conv_in_place(int64_t B, int64_t S, int64_t H, int E, int taps) {
  if (H % 16 != 0) return false;
  auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  const int64_t cols = up(E, 128), sms = num_sms();
  const int64_t in_place = up(B * up(S, 128) * cols, sms) * taps * up(H, 64);
  const int64_t unfolded = up(up(B * S, 128) * cols, sms) * up(taps * H, 64);
  return in_place - unfolded <= 22 + B * S * taps * H * 2 / 1900000;
}

size_t b200moe_conv_router_fwd_ws_bytes(int64_t B, int64_t S, int64_t H, int E, int taps) {
  if (B <= 0 || S <= 0 || H <= 0 || E <= 0 || taps <= 0 || conv_in_place(B, S, H, E, taps)) return 0;
  Carver c(nullptr);
  c.take<bf16_t>(B * S * taps * H);
  c.take<bf16_t>(static_cast<int64_t>(E) * taps * H);
  return c.off;
}

static int check_conv_router(const char* who, int64_t B, int64_t S, int64_t H, int E, int taps) {
  B200_CHECK_ARG(B > 0 && S > 0 && taps >= 1 && taps <= 64 && H > 0 && H % 8 == 0 && E > 0 && E % 8 == 0 && B * S < (1LL << 31),
                 B200MOE_E_BAD_SHAPE, "%s: B = %lld, S = %lld, H = %lld, E = %d (multiples of 8), taps = %d (1..64)", who,
                 (long long)B, (long long)S, (long long)H, E, taps);
  return 0;
}

int b200moe_conv_router_forward(const void* x, const void* weight, const float* bias, int64_t B, int64_t S, int64_t H, int E,
                                int taps, int k, int norm_topk, float scale, void* ws, void* weight_rows, void* logits,
                                int64_t* idx, float* w, int32_t* counts, int32_t* status, b200moe_stream_t stream) {
  int rc = check_conv_router("conv_router_forward", B, S, H, E, taps);
  if (rc) return rc;
  const bool in_place = conv_in_place(B, S, H, E, taps);
  B200_CHECK_ARG(x && weight && weight_rows && logits && (ws || in_place), B200MOE_E_NULL, "conv_router_forward: null pointer");
  RUN("conv_weight_rows", 1, conv_weight_rows(weight, E, H, taps, 0, weight_rows, counts, stream));
  if (in_place) {
    RUN("conv_gemm_logits", 1, b200moe_conv_gemm_logits(x, weight_rows, logits, B, S, H, E, taps, status, stream));
  } else {
    Carver c(ws);
    bf16_t* xu = c.take<bf16_t>(B * S * taps * H);
    bf16_t* wf = c.take<bf16_t>(static_cast<int64_t>(E) * taps * H);
    RUN("conv_weight_rows", 1, b200moe_conv_weight_rows(weight, E, H, taps, 1, wf, stream));
    RUN("conv_unfold", 1, b200moe_conv_unfold(x, B, S, H, taps, xu, stream));
    RUN("gemm_nt", 1, b200moe_gemm_nt(xu, wf, logits, B * S, E, taps * H, status, stream));
  }
  RUN("router_topk_fwd", 1, router_topk_fwd(logits, B200MOE_LOGITS_BF16, bias, B * S, E, k, norm_topk, scale, idx, w, counts, true, stream));
  return 0;
}

struct ConvBackward { bf16_t* u; float* part; };
static ConvBackward carve_conv(int64_t T, int64_t H, int64_t rows, void* ws, size_t* bytes) {
  Carver c(ws);
  ConvBackward b;
  b.u = c.take<bf16_t>(T * rows);
  b.part = c.take<float>(conv_split(T, rows, H, num_sms()).slices * rows * H);
  if (bytes != nullptr) *bytes = c.off;
  return b;
}

size_t b200moe_conv_router_bwd_ws_bytes(int64_t B, int64_t S, int64_t H, int E, int taps) {
  if (B <= 0 || S <= 0 || H <= 0 || E <= 0 || taps <= 0) return 0;
  size_t n = 0;
  carve_conv(B * S, H, static_cast<int64_t>(E) * taps, nullptr, &n);
  return n;
}

int b200moe_conv_router_backward(const void* x, const void* weight_rows, const void* logits, const int64_t* idx,
                                 const float* grad_w, int64_t B, int64_t S, int64_t H, int E, int taps, int k, int norm_topk,
                                 float scale, void* ws, void* grad_x, void* grad_weight, int32_t* status,
                                 b200moe_stream_t stream) {
  int rc = check_conv_router("conv_router_backward", B, S, H, E, taps);
  if (rc) return rc;
  B200_CHECK_ARG(x && weight_rows && ws, B200MOE_E_NULL, "conv_router_backward: null pointer");
  const int64_t T = B * S, rows = static_cast<int64_t>(E) * taps;
  const ConvBackward b = carve_conv(T, H, rows, ws, nullptr);
  RUN("conv_topk_bwd", 1, b200moe_conv_topk_bwd(logits, idx, grad_w, B, S, E, taps, k, norm_topk, scale, b.u, stream));
  if (grad_x != nullptr) RUN("gemm_nn", 1, b200moe_gemm_nn(b.u, weight_rows, grad_x, T, H, rows, status, stream));
  if (grad_weight != nullptr) {
    const Split sp = conv_split(T, rows, H, gemm_cta_budget());
    RUN("gemm_tn_splitk", 1, b200moe_gemm_tn_splitk(b.u, x, b.part, rows, H, T, sp.chunk, status, stream));
    RUN("conv_weight_grad", 1, b200moe_conv_weight_grad(b.part, sp.slices, E, H, taps, grad_weight, stream));
  }
  return 0;
}

// ---------------------------------------------------------------------------- experts on given picks
size_t b200moe_moe_fwd_ws_bytes(int64_t T, int64_t H, int64_t I, int E, int n_glu, int k, int keep, int row_kernels) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || k <= 0) return 0;
  size_t n = 0;
  carve_forward(make_dims(T, H, I, E, n_glu, k, keep, row_kernels), false, nullptr, &n);
  return n;
}

int b200moe_moe_forward(const void* x, const int64_t* idx, const float* w, const void* gate_up_proj, const void* down_proj,
                        const int32_t* act_codes, const float* act_params, int64_t T, int64_t H, int64_t I, int E, int n_glu,
                        int k, int keep, int row_kernels, void* ws, void* out, int32_t* status, b200moe_stream_t stream) {
  const Dims d = make_dims(T, H, I, E, n_glu, k, keep, row_kernels);
  int rc = check_dims("moe_forward", d);
  if (rc) return rc;
  B200_CHECK_ARG(x && idx && w && gate_up_proj && down_proj && ws && out, B200MOE_E_NULL, "moe_forward: null pointer");
  const Forward f = carve_forward(d, false, ws, nullptr);
  rc = permute(d, idx, f, nullptr, nullptr, status, stream);
  if (rc) return rc;
  return experts_forward(d, x, w, gate_up_proj, down_proj, act_codes, act_params, f, out, status, stream);
}

size_t b200moe_moe_bwd_ws_bytes(int64_t T, int64_t H, int64_t I, int E, int n_glu, int k, int row_kernels) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || k <= 0) return 0;
  size_t n = 0;
  carve_backward(make_dims(T, H, I, E, n_glu, k, 1, row_kernels), false, nullptr, &n);
  return n;
}

int b200moe_moe_backward(const void* grad_out, const float* w, const void* gate_up_proj, const void* down_proj,
                         const int32_t* act_codes, const float* act_params, int64_t T, int64_t H, int64_t I, int E,
                         int n_glu, int k, int row_kernels, void* fwd_ws, void* ws, void* grad_x, float* grad_w,
                         void* grad_gate_up, void* grad_down, float* grad_params, int32_t* status, b200moe_stream_t stream) {
  const Dims d = make_dims(T, H, I, E, n_glu, k, 1, row_kernels);
  int rc = check_dims("moe_backward", d);
  if (rc) return rc;
  B200_CHECK_ARG(grad_out && w && gate_up_proj && down_proj && fwd_ws && ws && grad_w, B200MOE_E_NULL, "moe_backward: null pointer");
  const Forward f = carve_forward(d, false, fwd_ws, nullptr);
  const Backward b = carve_backward(d, false, ws, nullptr);
  const Grads g{grad_x, grad_gate_up, grad_down, grad_w, grad_params};
  rc = experts_backward(d, grad_out, w, gate_up_proj, down_proj, act_codes, act_params, f, b, g, status, stream);
  if (rc) return rc;
  if (grad_x != nullptr) RUN("combine", 1, combine_add(b.grad_x_s, d.ldh(), nullptr, f.slot_row, nullptr, T, k, H, grad_x, stream));
  return 0;
}

// ---------------------------------------------------------------------------- router and experts
size_t b200moe_layer_fwd_ws_bytes(int64_t T, int64_t H, int64_t I, int E, int k, int keep) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || k <= 0) return 0;
  size_t n = 0;
  carve_forward(make_dims(T, H, I, E, E, k, keep, 0), true, nullptr, &n);
  return n;
}

int b200moe_layer_forward(const void* x, const void* gate_weight, const float* bias, const void* gate_up_proj,
                          const void* down_proj, const int32_t* act_codes, int64_t T, int64_t H, int64_t I, int E, int k,
                          int norm_topk, float scale, int keep, void* ws, int32_t* counts, int64_t* load, void* out,
                          int32_t* status, b200moe_stream_t stream) {
  const Dims d = make_dims(T, H, I, E, E, k, keep, 0);
  int rc = check_dims("layer_forward", d);
  if (rc) return rc;
  B200_CHECK_ARG(x && gate_weight && gate_up_proj && down_proj && ws && out, B200MOE_E_NULL, "layer_forward: null pointer");
  const Forward f = carve_forward(d, true, ws, nullptr);
  rc = router_forward(x, gate_weight, bias, T, H, E, k, norm_topk, scale, f.logits, f.idx, f.w, nullptr, status, stream);
  if (rc) return rc;
  rc = permute(d, f.idx, f, counts, load, status, stream);
  if (rc) return rc;
  return experts_forward(d, x, f.w, gate_up_proj, down_proj, act_codes, nullptr, f, out, status, stream);
}

size_t b200moe_layer_bwd_ws_bytes(int64_t T, int64_t H, int64_t I, int E, int k) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || k <= 0) return 0;
  size_t n = 0;
  carve_backward(make_dims(T, H, I, E, E, k, 1, 0), true, nullptr, &n);
  return n;
}

int b200moe_layer_backward(const void* grad_out, const void* x, const void* gate_weight, const void* gate_up_proj,
                           const void* down_proj, const int32_t* act_codes, int64_t T, int64_t H, int64_t I, int E, int k,
                           int norm_topk, float scale, void* fwd_ws, void* ws, void* grad_x, void* grad_gate_weight,
                           void* grad_gate_up, void* grad_down, int32_t* status, b200moe_stream_t stream) {
  const Dims d = make_dims(T, H, I, E, E, k, 1, 0);
  int rc = check_dims("layer_backward", d);
  if (rc) return rc;
  B200_CHECK_ARG(grad_out && x && gate_weight && gate_up_proj && down_proj && fwd_ws && ws, B200MOE_E_NULL, "layer_backward: null pointer");
  const Forward f = carve_forward(d, true, fwd_ws, nullptr);
  const Backward b = carve_backward(d, true, ws, nullptr);
  const Grads g{grad_x, grad_gate_up, grad_down, b.grad_w, nullptr};
  rc = experts_backward(d, grad_out, f.w, gate_up_proj, down_proj, act_codes, nullptr, f, b, g, status, stream);
  if (rc) return rc;
  if (grad_x != nullptr || grad_gate_weight != nullptr) {
    rc = router_backward(x, gate_weight, f.logits, f.idx, b.grad_w, T, H, E, k, norm_topk, scale, b.grad_logits, b.part,
                         grad_x != nullptr ? b.grad_x_router : nullptr, grad_gate_weight, status, stream);
    if (rc) return rc;
  }
  if (grad_x != nullptr)   // the experts' rows of a token and the router's share, added in fp32, one rounding
    RUN("combine", 1, combine_add(b.grad_x_s, d.ldh(), nullptr, f.slot_row, b.grad_x_router, T, k, H, grad_x, stream));
  return 0;
}

// ---------------------------------------------------------------------------- Newton-Schulz iterations
// The segments are padded to Rp rows for the GEMM's row tiles; only the first `rows_live` (rounded up to 64) of them carry
// anything, so the Gram matrices are neither computed nor read past that column.  Their pad rows past it then hold whatever
// the buffers held: they meet nothing but pad rows of the results.  (The step over stacks of 64 x 2816 x 2048, without padding, and
// 64 x 1408 x 2048, Rp 1536: 20 products X X^T 9.97 -> 9.63 ms, b A + c A A 8.39 -> 7.98, B X 16.85 -> 16.05.)
int b200moe_newton_schulz(void* x, void* x_next, void* a, void* a2, const int32_t* tile_expert, const int32_t* poffs, int E,
                          int64_t Rp, int64_t rows_live, int64_t wide, const float* coeffs, int iterations, int32_t* status,
                          b200moe_stream_t stream) {
  B200_CHECK_ARG(x && x_next && a && a2 && coeffs, B200MOE_E_NULL, "newton_schulz: null pointer");
  B200_CHECK_ARG(iterations >= 0 && rows_live >= 1 && rows_live <= Rp && Rp - rows_live < 256, B200MOE_E_BAD_SHAPE,
                 "newton_schulz: iterations = %d, %lld of Rp = %lld rows live", iterations, (long long)rows_live, (long long)Rp);
  const int64_t rows = E * Rp, live = (rows_live + 63) / 64 * 64;
  for (int i = 0; i < iterations; ++i) {
    const float ca = coeffs[3 * i], cb = coeffs[3 * i + 1], cc = coeffs[3 * i + 2];
    RUN("expert_gram", 1, expert_gram(x, tile_expert, poffs, rows, E, wide, 1, live, a, status, stream));
    RUN("expert_linear_axpby", 1, expert_linear_axpby(a, a, a, cc, cb, ca, 2, tile_expert, poffs, rows, E, Rp, Rp, live, live, a2, status, stream));
    RUN("expert_linear_t", 1, expert_linear_t(a2, Rp, x, tile_expert, poffs, rows, E, Rp, wide, live, x_next, wide, status, stream));
    std::swap(x, x_next);
  }
  return 0;
}

}  // extern "C"
