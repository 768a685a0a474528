// Router epilogue kernels: sigmoid + selection bias + in-register warp-level top-k + renormalise
// (forward), the matching Jacobian (backward), the bias update and the split-K slice reduction.
// One warp owns one token; lane l holds experts l, l+32, ... (at most 8 values for E <= 256).
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"
#include "topk.cuh"

namespace b200moe {


template <int KIND>
__device__ __forceinline__ float load_in(const void* p, long long i) {
  if (KIND == B200MOE_LOGITS_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}

// Both kernels are bound by instruction issue and by the latency of the k dependent picks, not by their few bytes per
// token.  VPL = values per lane = ceil(E / 32) rounded up to a power of two: compiled per width, since a fixed VPL of 8
// spends its compares on experts that do not exist (T = 16384, E = 64, k = 6: 23.9 -> 10.5 us; T = 32768, E = 128,
// k = 8: 80 -> 26 us).  A pick is one
// redux.max over the lanes' best keys and one redux.min over the ids that hold it (ties to the lowest expert id, as a
// stable sort gives), instead of five shuffle rounds of (value, id) pairs.
template <int KIND, int VPL>
__global__ void __launch_bounds__(256)
router_topk_fwd_kernel(const void* input, const float* bias, long long T, int E, int k, int norm, float scale,
                       long long* idx_out, float* w_out, int* counts) {
  grid_dep_begin();
  __shared__ int hist[B200MOE_MAX_EXPERTS];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  for (int e = threadIdx.x; e < E; e += blockDim.x) hist[e] = 0;
  __syncthreads();

  float b[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int e = lane + 32 * i;
    b[i] = (bias != nullptr && e < E) ? bias[e] : 0.0f;
  }

  for (long long t = static_cast<long long>(blockIdx.x) * wpb + warp; t < T;
       t += static_cast<long long>(gridDim.x) * wpb) {
    float sc[VPL];
    uint32_t key[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int e = lane + 32 * i;
      sc[i] = 0.0f;
      key[i] = 0u;
      if (e < E) {
        const float v = load_in<KIND>(input, t * E + e);
        sc[i] = (KIND == B200MOE_SCORES_F32) ? v : sigmoid_f(v);
        key[i] = select_key(sc[i] + b[i]);
      }
    }
    int my_idx;
    float my_w;
    topk_of_token<VPL>(sc, key, k, norm, scale, hist, counts != nullptr, my_idx, my_w);
    if (lane < k) {
      idx_out[t * k + lane] = my_idx;
      w_out[t * k + lane] = my_w;
    }
  }
  if (counts != nullptr) {
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
      const int c = hist[e];
      if (c != 0) atomicAdd(&counts[e], c);
    }
  }
}

// taps > 1 (the conv router; rows are (batch, position), S positions): grad_logits is written as the operand of the
// products for dX and dW, u (T, taps*E), u[s', j*E + e] = grad_logits[s' + (taps-1) - j, e], zero past the end.
// Lane j < k reads pick j, its upstream gradient and its logit, so the dependent loads of all picks are one round trip;
// the sums run over the picks in order.  (T = 16384, E = 64, k = 6: 14.2 -> 6.8 us.)
template <int KIND, int VPL, bool PAIR>
__global__ void __launch_bounds__(256)
router_topk_bwd_kernel(const void* logits, const long long* idx, const float* grad_w, long long T, int E, int k,
                       int norm, float scale, int S, int taps, __nv_bfloat16* grad_logits) {
  grid_dep_begin();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  // expert of a lane's i-th value; PAIR (even E): neighbours two by two, so that a warp writes whole 32-bit words
  auto expert = [lane](int i) { return PAIR ? 64 * (i >> 1) + 2 * lane + (i & 1) : lane + 32 * i; };
  for (long long t = static_cast<long long>(blockIdx.x) * wpb + warp; t < T;
       t += static_cast<long long>(gridDim.x) * wpb) {
    float s[VPL], gs[VPL];
    int ik = -1;
    float gk = 0.0f, wk = 0.0f;
    if (lane < k) {
      ik = static_cast<int>(idx[t * k + lane]);
      gk = grad_w[t * k + lane];
    }
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int e = expert(i);
      s[i] = (e < E) ? sigmoid_f(load_in<KIND>(logits, t * E + e)) : 0.0f;
      gs[i] = 0.0f;
    }
    float graw = gk * scale;
    if (norm && k > 1) {
      if (ik >= 0 && ik < E) wk = sigmoid_f(load_in<KIND>(logits, t * E + ik));
      float tsum = 0.0f, dot = 0.0f;
      const float gw = gk * wk;
      for (int j = 0; j < k; ++j) {
        tsum += __shfl_sync(0xffffffffu, wk, j);
        dot += __shfl_sync(0xffffffffu, gw, j);
      }
      tsum += 1e-20f;
      graw = (scale / tsum) * (gk - dot / tsum);
    }
    for (int j = 0; j < k; ++j) {
      const int ij = __shfl_sync(0xffffffffu, ik, j);
      const float gj = __shfl_sync(0xffffffffu, graw, j);
#pragma unroll
      for (int i = 0; i < VPL; ++i)
        if (ij == expert(i)) gs[i] += gj;
    }
    auto put = [&](long long row, const uint32_t (&g)[VPL]) {     // g: bf16 bits of this lane's values
#pragma unroll
      for (int i = 0; i < VPL; i += PAIR ? 2 : 1) {
        const int e = expert(i);
        if (e >= E) continue;
        if constexpr (PAIR) *reinterpret_cast<uint32_t*>(grad_logits + row * E + e) = g[i] | (g[i + 1] << 16);
        else reinterpret_cast<uint16_t*>(grad_logits)[row * E + e] = static_cast<uint16_t>(g[i]);
      }
    };
    uint32_t g[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) g[i] = pack_bf16x2(gs[i] * (s[i] * (1.0f - s[i])), 0.0f);
    if (taps == 1) {
      put(t, g);
      continue;
    }
    const uint32_t zero[VPL] = {};
    const int pos = static_cast<int>(t % S);
    for (int j = 0; j < taps; ++j) {
      const int back = taps - 1 - j;       // this token's gradient belongs to the row `back` positions earlier
      if (pos >= back) put((t - back) * taps + j, g);
      if (pos + back >= S) put(t * taps + j, zero);
    }
  }
}

// w (E, H, taps) -> wt (taps, E, H), wt[j, e, h] = w[e, h, j] (the operand of the conv router's products), or (E, taps, H).  counts (E,
// nullable) are cleared for the top-k kernel further on: a memset between the two would end their chain of launches (5 us).
__global__ void __launch_bounds__(256)
conv_weight_rows_kernel(const __nv_bfloat16* w, int E, int H, int taps, int by_expert, __nv_bfloat16* wt, int* counts) {
  grid_dep_begin();
  if (counts != nullptr && blockIdx.x == 0)
    for (int e = threadIdx.x; e < E; e += 256) counts[e] = 0;
  const long long n = static_cast<long long>(E) * H;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
    const long long e = i / H, h = i - e * H;
    for (int j = 0; j < taps; ++j)
      wt[(by_expert ? e * taps + j : static_cast<long long>(j) * E + e) * H + h] = w[i * taps + j];
  }
}

// grad_w (E, H, taps) bf16 = sum over the slices of p (slices, taps*E, H) fp32
__global__ void __launch_bounds__(256)
conv_weight_grad_kernel(const float* p, long long slices, int E, int H, int taps, __nv_bfloat16* gw) {
  grid_dep_begin();
  const long long n = static_cast<long long>(E) * H, elems = n * taps;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < elems; i += gridDim.x * 256LL) {
    const long long j = i / n, eh = i - j * n;       // consecutive threads: consecutive h of one row of p
    float acc = 0.0f;
#pragma unroll 8
    for (long long q = 0; q < slices; ++q) acc += p[q * elems + i];
    gw[eh * taps + j] = __float2bfloat16_rn(acc);
  }
}

__global__ void router_bias_update_kernel(float* bias, const int* counts, int E, float u) {
  __shared__ float red[32];
  float part = 0.0f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) part += static_cast<float>(counts[e]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  __syncthreads();
  float total = 0.0f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) total += red[i];
  const float mean = total / static_cast<float>(E);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float d = mean - static_cast<float>(counts[e]);
    const float sg = (d > 0.0f) ? 1.0f : (d < 0.0f ? -1.0f : 0.0f);
    bias[e] += u * sg;
  }
}

// D[i] = bf16( sum_s P[s][i] ), 4 elements per thread
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* P, long long slices, long long elems, __nv_bfloat16* D) {
  grid_dep_begin();
  const long long i4 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (i4 >= elems) return;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long long s = 0; s < slices; ++s) {
    const float4 v = *reinterpret_cast<const float4*>(P + s * elems + i4);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  uint2 o;
  o.x = pack_bf16x2(acc.x, acc.y);
  o.y = pack_bf16x2(acc.z, acc.w);
  *reinterpret_cast<uint2*>(D + i4) = o;
}

// D (C,R) = bf16( sum_s P[s] (R,C) )^T through a 32 x 32 tile in shared memory: both sides coalesced, a thread per
// value so that all its slices are in flight at once
__global__ void __launch_bounds__(1024)
splitk_reduce_t_kernel(const float* P, long long slices, int R, int C, __nv_bfloat16* D) {
  grid_dep_begin();
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const long long elems = static_cast<long long>(R) * C;
  float acc = 0.0f;
  if (r0 + ty < R && c0 + tx < C) {
    const float* src = P + static_cast<long long>(r0 + ty) * C + c0 + tx;
#pragma unroll 16
    for (long long s = 0; s < slices; ++s) acc += src[s * elems];
  }
  tile[ty][tx] = acc;
  __syncthreads();
  if (r0 + tx < R && c0 + ty < C) D[static_cast<long long>(c0 + ty) * R + r0 + tx] = __float2bfloat16_rn(tile[tx][ty]);
}

static int grid_for_tokens(long long T) {
  long long g = (T + 7) / 8;
  const long long cap = static_cast<long long>(num_sms()) * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

template <int KIND>
static cudaError_t launch_topk_bwd(const void* logits, const long long* idx, const float* grad_w, long long T, int E, int k, int norm,
                            float scale, int S, int taps, __nv_bfloat16* out, cudaStream_t st) {
  const int grid = grid_for_tokens(T);
  cudaError_t err = cudaSuccess;
  by_experts(E, [&](auto v) {
    constexpr int VPL = v.value;
    const bool pair = VPL > 1 && E % 2 == 0 && reinterpret_cast<uintptr_t>(out) % 4 == 0;
    err = launch_chained(pair ? router_topk_bwd_kernel<KIND, VPL, (VPL > 1)> : router_topk_bwd_kernel<KIND, VPL, false>, grid, 256, 0,
                         st, 1, logits, idx, grad_w, T, E, k, norm, scale, S, taps, out);
  });
  return err;
}

static int weight_grid(int64_t n) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, static_cast<int64_t>(num_sms()) * 8)));
}

int conv_weight_rows(const void* w, int E, int64_t H, int taps, int by_expert, void* wt, int32_t* counts, b200moe_stream_t stream) {
  B200_CHECK_ARG(w && wt, B200MOE_E_NULL, "conv_weight_rows: null pointer");
  B200_CHECK_ARG(E >= 1 && H >= 1 && H < (1LL << 31) && taps >= 1, B200MOE_E_BAD_SHAPE, "conv_weight_rows: E = %d, H = %lld, taps = %d", E,
                 (long long)H, taps);
  B200_LAUNCH(conv_weight_rows_kernel, weight_grid(E * H), 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(w), E,
              static_cast<int>(H), taps, by_expert, reinterpret_cast<__nv_bfloat16*>(wt), counts);
  return 0;
}

int router_topk_fwd(const void* input, int input_kind, const float* bias, int64_t T, int E, int k, int norm_topk, float scale, int64_t* idx,
                    float* w, int32_t* counts, bool counts_cleared, b200moe_stream_t stream) {
  B200_CHECK_ARG(input && idx && w, B200MOE_E_NULL, "router_topk_fwd: null pointer");
  B200_CHECK_ARG(E >= 1 && E <= B200MOE_MAX_EXPERTS, B200MOE_E_UNSUPPORTED,
                 "router_topk_fwd: E = %d, supported 1..%d", E, B200MOE_MAX_EXPERTS);
  B200_CHECK_ARG(k >= 1 && k <= E && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE,
                 "router_topk_fwd: top_k = %d must be in 1..min(E=%d, %d)", k, E, B200MOE_MAX_TOPK);
  B200_CHECK_ARG(T >= 0, B200MOE_E_BAD_SHAPE, "router_topk_fwd: T = %lld", (long long)T);
  cudaStream_t st = (cudaStream_t)stream;
  if (counts != nullptr && !counts_cleared) B200_CUDA(cudaMemsetAsync(counts, 0, sizeof(int32_t) * E, st));
  if (T == 0) return 0;
  const int grid = grid_for_tokens(T);
  long long* idx_ll = reinterpret_cast<long long*>(idx);
  cudaError_t err = cudaSuccess;
  switch (input_kind) {
    case B200MOE_LOGITS_BF16:
      by_experts(E, [&](auto v) { err = launch_chained(router_topk_fwd_kernel<B200MOE_LOGITS_BF16, v.value>, grid, 256, 0, st, 1, input, bias, T, E, k, norm_topk, scale, idx_ll, w, counts); });
      break;
    case B200MOE_LOGITS_F32:
      by_experts(E, [&](auto v) { err = launch_chained(router_topk_fwd_kernel<B200MOE_LOGITS_F32, v.value>, grid, 256, 0, st, 1, input, bias, T, E, k, norm_topk, scale, idx_ll, w, counts); });
      break;
    case B200MOE_SCORES_F32:
      by_experts(E, [&](auto v) { err = launch_chained(router_topk_fwd_kernel<B200MOE_SCORES_F32, v.value>, grid, 256, 0, st, 1, input, bias, T, E, k, norm_topk, scale, idx_ll, w, counts); });
      break;
    default:
      set_error("router_topk_fwd: unknown input_kind %d", input_kind);
      return B200MOE_E_UNSUPPORTED;
  }
  B200_CUDA(err);
  return 0;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_router_topk_fwd(const void* input, int input_kind, const float* bias, int64_t T, int E, int k,
                            int norm_topk, float scale, int64_t* idx, float* w, int32_t* counts,
                            b200moe_stream_t stream) {
  return router_topk_fwd(input, input_kind, bias, T, E, k, norm_topk, scale, idx, w, counts, false, stream);
}

int b200moe_router_topk_bwd(const void* logits, int input_kind, const int64_t* idx, const float* grad_w, int64_t T,
                            int E, int k, int norm_topk, float scale, void* grad_logits, b200moe_stream_t stream) {
  B200_CHECK_ARG(logits && idx && grad_w && grad_logits, B200MOE_E_NULL, "router_topk_bwd: null pointer");
  B200_CHECK_ARG(E >= 1 && E <= B200MOE_MAX_EXPERTS, B200MOE_E_UNSUPPORTED,
                 "router_topk_bwd: E = %d, supported 1..%d", E, B200MOE_MAX_EXPERTS);
  B200_CHECK_ARG(k >= 1 && k <= E && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE, "router_topk_bwd: top_k = %d", k);
  if (T <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const long long* idx_ll = reinterpret_cast<const long long*>(idx);
  __nv_bfloat16* gl = reinterpret_cast<__nv_bfloat16*>(grad_logits);
  switch (input_kind) {
    case B200MOE_LOGITS_BF16:
      B200_CUDA(launch_topk_bwd<B200MOE_LOGITS_BF16>(logits, idx_ll, grad_w, T, E, k, norm_topk, scale, 1, 1, gl, st));
      break;
    case B200MOE_LOGITS_F32:
      B200_CUDA(launch_topk_bwd<B200MOE_LOGITS_F32>(logits, idx_ll, grad_w, T, E, k, norm_topk, scale, 1, 1, gl, st));
      break;
    default:
      set_error("router_topk_bwd: input_kind %d has no backward (logits are required)", input_kind);
      return B200MOE_E_UNSUPPORTED;
  }
  return 0;
}

int b200moe_conv_topk_bwd(const void* logits, const int64_t* idx, const float* grad_w, int64_t B, int64_t S, int E, int taps,
                          int k, int norm_topk, float scale, void* u, b200moe_stream_t stream) {
  B200_CHECK_ARG(logits && idx && grad_w && u, B200MOE_E_NULL, "conv_topk_bwd: null pointer");
  B200_CHECK_ARG(E >= 1 && E <= B200MOE_MAX_EXPERTS, B200MOE_E_UNSUPPORTED, "conv_topk_bwd: E = %d, supported 1..%d", E,
                 B200MOE_MAX_EXPERTS);
  B200_CHECK_ARG(k >= 1 && k <= E && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE, "conv_topk_bwd: top_k = %d", k);
  B200_CHECK_ARG(B >= 1 && S >= 1 && S < (1LL << 31) && taps >= 1 && taps <= 64, B200MOE_E_BAD_SHAPE,
                 "conv_topk_bwd: B = %lld, S = %lld, taps = %d (1..64)", (long long)B, (long long)S, taps);
  B200_CUDA(launch_topk_bwd<B200MOE_LOGITS_BF16>(logits, reinterpret_cast<const long long*>(idx), grad_w, B * S, E, k, norm_topk,
                                                 scale, static_cast<int>(S), taps, reinterpret_cast<__nv_bfloat16*>(u),
                                                 (cudaStream_t)stream));
  return 0;
}

int b200moe_conv_weight_rows(const void* w, int E, int64_t H, int taps, int by_expert, void* wt, b200moe_stream_t stream) {
  return conv_weight_rows(w, E, H, taps, by_expert, wt, nullptr, stream);
}

int b200moe_conv_weight_grad(const float* P, int64_t slices, int E, int64_t H, int taps, void* grad_w,
                             b200moe_stream_t stream) {
  B200_CHECK_ARG(P && grad_w, B200MOE_E_NULL, "conv_weight_grad: null pointer");
  B200_CHECK_ARG(slices >= 1 && E >= 1 && H >= 1 && H < (1LL << 31) && taps >= 1, B200MOE_E_BAD_SHAPE,
                 "conv_weight_grad: slices = %lld, E = %d, H = %lld, taps = %d", (long long)slices, E, (long long)H, taps);
  B200_LAUNCH(conv_weight_grad_kernel, weight_grid(E * H * taps), 256, 0, stream, P, slices, E, static_cast<int>(H), taps,
              reinterpret_cast<__nv_bfloat16*>(grad_w));
  return 0;
}

int b200moe_router_bias_update(float* bias, const int32_t* counts, int E, float u, b200moe_stream_t stream) {
  B200_CHECK_ARG(bias && counts, B200MOE_E_NULL, "router_bias_update: null pointer");
  B200_CHECK_ARG(E >= 1, B200MOE_E_BAD_SHAPE, "router_bias_update: E = %d", E);
  if (!(u > 0.0f)) return 0;
  router_bias_update_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(bias, counts, E, u);
  B200_CUDA(cudaGetLastError());
  return 0;
}

int b200moe_splitk_reduce_t(const float* P, int64_t slices, int64_t R, int64_t C, void* D, b200moe_stream_t stream) {
  B200_CHECK_ARG(P && D, B200MOE_E_NULL, "splitk_reduce_t: null pointer");
  B200_CHECK_ARG(slices >= 1 && R > 0 && C > 0 && R < (1LL << 31) && C <= 32 * 65535, B200MOE_E_BAD_SHAPE,
                 "splitk_reduce_t: slices = %lld, R = %lld, C = %lld", (long long)slices, (long long)R, (long long)C);
  const dim3 grid(static_cast<unsigned>((R + 31) / 32), static_cast<unsigned>((C + 31) / 32));
  B200_LAUNCH(splitk_reduce_t_kernel, grid, 1024, 0, stream, P, slices, static_cast<int>(R), static_cast<int>(C),
              reinterpret_cast<__nv_bfloat16*>(D));
  return 0;
}

int b200moe_splitk_reduce(const float* P, int64_t slices, int64_t elems, void* D, b200moe_stream_t stream) {
  B200_CHECK_ARG(P && D, B200MOE_E_NULL, "splitk_reduce: null pointer");
  B200_CHECK_ARG(slices >= 1 && elems > 0 && elems % 4 == 0, B200MOE_E_BAD_SHAPE,
                 "splitk_reduce: slices = %lld, elems = %lld (must be a multiple of 4)", (long long)slices,
                 (long long)elems);
  const long long threads = elems / 4;
  const int grid = static_cast<int>((threads + 255) / 256);
  B200_LAUNCH(splitk_reduce_kernel, grid, 256, 0, stream, P, slices, elems, reinterpret_cast<__nv_bfloat16*>(D));
  return 0;
}

}  // extern "C"
