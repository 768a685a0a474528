// PolyGLU activations with a per-expert activation code, as separate row kernels (the path used when
// an expert stack is not pure SiLU-GLU; the pure stack runs fused in the GEMM epilogues).
//   codes: 0 SiLU, 1 ReLU^2, 2 NormSiLU, 5 SiTU (gamma * tanh(alpha g) * sigmoid(g)), 6 NormReLU^2,
//          7 NormSiTU; the Norm codes first divide the gate row by rms = sqrt(mean(g^2) + 1e-6).
//   codes 3 (Identity) and 4 (Zero) are expert KINDS without weights: their rows are copied / zeroed.
// Semantics follow kernels/sm75/moe.py:163-232 (_glu_fwd_row_kernel, _glu_bwd_row_kernel) and
// :859-881 (_act_eager) of the reference; math in fp32, bf16 in and out.
//
// Bound: HBM (forward 3 I, backward 5 I bf16 values a row) and, close behind it, the instructions of the activations.  The kernels that
// carry the path (`glu_*_vec_kernel`) hold a row in registers: TPR threads share a row, each with VPT 16-byte vectors of
// every operand, all loaded before the first use, so a row is read once however many reductions its activation needs.
// Rows of one CTA lie inside one 256-row tile and share its expert, so the activation code is uniform over the CTA and
// the element loops are compiled per code.  The one-value-per-thread kernels below them read each value with a
// 2-byte access, once per reduction; they remain for d_ff that is no multiple of 8 or above 8192 and for unaligned
// buffers.  32 768 rows, codes 0 1 2 5 6 7 in turn, L2 flushed before, dense rows, us (at copy rate): d_ff 768 forward 37 (25), backward 59
// (41); d_ff 1032 57 (33), 100 (55); 8192 rows of d_ff 4096 47 (31), 74 (52).  With divisions, rows of 64 x 2 and 128 x 2 vectors, and the
// Norm codes' activations kept across the second reduction they took 51 / 96, 86 / 170 and 59 / 103.  1 - sigmoid and 1 - tanh^2 as differences: backward
// 55, 107 and 72.
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace b200moe {

constexpr float kRmsEps = 1e-6f;   // _NS_EPS, kernels/sm75/moe.py:80

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.0f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) s += red[i];
  return s;
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float tanh_via_sigmoid(float x) { return 2.0f / (1.0f + expf(-2.0f * x)) - 1.0f; }
__device__ __forceinline__ bool is_norm(int code) { return code == 2 || code == 6 || code == 7; }

// activation value f(gn) (times gamma for SiTU) for the forward; gn = gate or gate / rms
__device__ __forceinline__ float act_value(int code, float gate, float gn, float alpha, float gamma) {
  const float sig = sigmoidf_(gn);
  if (code == 1 || code == 6) {
    const float r = fmaxf(gn, 0.0f);
    return r * r;
  }
  if (code == 5) return gamma * tanh_via_sigmoid(alpha * gate) * sig;
  if (code == 7) return tanh_via_sigmoid(gn) * sig;
  return gn * sig;   // codes 0 and 2
}

// ---------------------------------------------------------------------------- a row held in registers
constexpr int kRowThreads = 256;

// sum over the TPR threads of a row; every thread of the CTA calls it (uniformly)
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if constexpr (TPR > 32) {
    const int warp = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[warp] = v;
    __syncthreads();
    const int w0 = warp & ~(TPR / 32 - 1);
    v = 0.0f;
#pragma unroll
    for (int i = 0; i < TPR / 32; ++i) v += red[w0 + i];
  }
  return v;
}

// Reciprocal of a number from 0.5 to 2 by the special-function unit, within one unit in the last place.  The correctly rounded division took
// more instructions than the exponential beside it (forward 53 -> 44 us, backward 98 -> 80 of 32 768 rows of d_ff 768, below).
__device__ __forceinline__ float rcp_near_1(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// activation value and its derivative with respect to gn (gn = gate, or gate / rms for the Norm codes).  Code 5:
// dal = d(act)/d(alpha), t5s = act / gamma
// Sigmoid and tanh from exponentials of -|x|, which lie in [0, 1]: sig and rest = 1 - sig are 1 / (1 + a) and a / (1 + a) or the other way
// round, 1 - tanh^2 is 4 b / (1 + b)^2.  As differences from 1 nothing is left of the former from gates of 16 on, of the latter from 8 on; and
// nothing overflows or is flushed.
template <int CODE>
__device__ __forceinline__ void act_eval(float gn, float alpha, float gamma, float& act, float& d, float& dal, float& t5s) {
  if constexpr (CODE == 1 || CODE == 6) {
    const float r = fmaxf(gn, 0.0f);
    act = r * r;
    d = 2.0f * r;
  } else {
    const float a = expf(-fabsf(gn)), r = rcp_near_1(1.0f + a), ar = a * r;
    const float sig = gn >= 0.0f ? r : ar;
    if constexpr (CODE == 5 || CODE == 7) {
      const float rest = gn >= 0.0f ? ar : r, x = CODE == 5 ? alpha * gn : gn;
      const float b = CODE == 5 ? expf(-2.0f * fabsf(x)) : a * a, h = rcp_near_1(0.5f + 0.5f * b);       // h = 2 / (1 + b)
      const float t = copysignf((0.5f - 0.5f * b) * h, x), dt = (b * h) * h;                          // tanh(x), 1 - tanh(x)^2
      const float gs = CODE == 5 ? gamma * sig : sig;
      act = gs * t;
      if constexpr (CODE == 5) {
        d = gs * (alpha * dt + t * rest);
        dal = gs * gn * dt;
        t5s = t * sig;
      } else {
        d = gs * (dt + t * rest);
      }
    } else {
      act = gn * sig;
      d = sig * (1.0f + gn * (1.0f - sig));        // (the difference is added to 1)
    }
  }
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

template <int TPR, int VPT>
__device__ __forceinline__ float row_rms_inv(const uint4 (&g)[VPT], int I, float* red) {
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    float f[8];
    unpack8(g[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = row_sum<TPR>(ss, red);
  return 1.0f / sqrtf(ss / static_cast<float>(I) + kRmsEps);
}

template <int CODE, int TPR, int VPT>
__device__ __forceinline__ void glu_fwd_row(const uint4 (&g)[VPT], const uint4 (&u)[VPT], uint4* dst, int t, int nvec,
                                            float alpha, float gamma, float* red) {
  constexpr bool NORM = CODE == 2 || CODE == 6 || CODE == 7;
  float inv_r = 1.0f;
  if constexpr (NORM) inv_r = row_rms_inv<TPR, VPT>(g, nvec * 8, red);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = t + TPR * i;
    if (c >= nvec) continue;
    float gf[8], uf[8];
    unpack8(g[i], gf);
    unpack8(u[i], uf);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float act, d, dal, t5s;
      act_eval<CODE>(NORM ? gf[j] * inv_r : gf[j], alpha, gamma, act, d, dal, t5s);
      gf[j] = act * uf[j];
    }
    dst[c] = pack8(gf);
  }
}

template <int TPR, int VPT>
__global__ void __launch_bounds__(kRowThreads)
glu_fwd_vec_kernel(const uint4* gate_up, const int* tile_expert, const int* codes, const float* params,
                   const int* total_rows, int nvec, int pitch2, uint4* inter, int pitch) {
  grid_dep_begin();
  constexpr int RPB = kRowThreads / TPR;   // rows a CTA works on at a time; divides the 256-row tile
  __shared__ float red[kRowThreads / 32];
  const int total = *total_rows;
  const int t = threadIdx.x % TPR;
  for (long long r0 = static_cast<long long>(blockIdx.x) * RPB; r0 < total; r0 += static_cast<long long>(gridDim.x) * RPB) {
    const long long r = r0 + threadIdx.x / TPR;
    const bool live = r < total;
    const int n = live ? nvec : 0;         // a row past the end takes part in the reductions with zeros
    uint4 g[VPT], u[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = t + TPR * i;
      g[i] = c < n ? gate_up[r * pitch2 + c] : make_uint4(0u, 0u, 0u, 0u);
      u[i] = c < n ? gate_up[r * pitch2 + nvec + c] : make_uint4(0u, 0u, 0u, 0u);
    }
    const int e = tile_expert[r0 / B200MOE_TILE_M];
    const int code = codes[e];
    const float alpha = (params != nullptr && code == 5) ? params[2 * e] : 1.0f;
    const float gamma = (params != nullptr && code == 5) ? params[2 * e + 1] : 1.0f;
    uint4* dst = inter + r * pitch;
    switch (code) {                        // uniform over the CTA
      case 1: glu_fwd_row<1, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
      case 2: glu_fwd_row<2, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
      case 5: glu_fwd_row<5, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
      case 6: glu_fwd_row<6, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
      case 7: glu_fwd_row<7, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
      default: glu_fwd_row<0, TPR, VPT>(g, u, dst, t, n, alpha, gamma, red); break;
    }
  }
}

// da / dg: this thread's share of the row's alpha / gamma gradient (code 5 only)
template <int CODE, int TPR, int VPT>
__device__ __forceinline__ void glu_bwd_row(const uint4 (&g)[VPT], const uint4 (&u)[VPT], const uint4 (&go)[VPT],
                                            uint4* gg, uint4* gu, int t, int nvec, float alpha, float gamma, float* red,
                                            float& da, float& dg) {
  constexpr bool NORM = CODE == 2 || CODE == 6 || CODE == 7;
  float inv_r = 1.0f, part = 0.0f;
  float wd[NORM ? VPT : 1][8];            // Norm codes: go * up * f'(gn), kept until the row's coupling term is known
  if constexpr (NORM) inv_r = row_rms_inv<TPR, VPT>(g, nvec * 8, red);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = t + TPR * i;
    float gf[8], uf[8], of[8];
    unpack8(g[i], gf);
    unpack8(u[i], uf);
    unpack8(go[i], of);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gn = NORM ? gf[j] * inv_r : gf[j];
      float act, d, dal = 0.0f, t5s = 0.0f;
      act_eval<CODE>(gn, alpha, gamma, act, d, dal, t5s);
      const float w = of[j] * uf[j];
      if constexpr (CODE == 5)
        if (c < nvec) {                    // an idle lane's zeros are NaN times an infinite parameter
          da += w * dal;
          dg += w * t5s;
        }
      uf[j] = of[j] * act;
      if constexpr (NORM) {
        wd[i][j] = w * d;
        part += wd[i][j] * gn;
      } else {
        gf[j] = w * d;
      }
    }
    if (c < nvec) {
      gu[c] = pack8(uf);
      if constexpr (!NORM) gg[c] = pack8(gf);
    }
  }
  if constexpr (NORM) {   // RMS coupling term: mean of go * up * f'(gn) * gn
    const float S = row_sum<TPR>(part, red) / static_cast<float>(nvec * 8);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = t + TPR * i;
      float gf[8];
      unpack8(g[i], gf);
#pragma unroll
      for (int j = 0; j < 8; ++j) gf[j] = (wd[i][j] - S * (gf[j] * inv_r)) * inv_r;
      if (c < nvec) gg[c] = pack8(gf);
    }
  }
}

// The register bounds hold three and two CTAs on an SM: left to itself the compiler took 87 registers for 32 x 2 vectors (32 768 rows of d_ff 256 36 -> 41
// us) and scheduled three vectors a thread worse (d_ff 768 59 -> 64, 1032 100 -> 113); four are better left alone (4096 rows of d_ff 8192 88 -> 82).
template <int TPR, int VPT>
__global__ void __launch_bounds__(kRowThreads, VPT == 2 ? 3 : VPT == 3 ? 2 : 0)
glu_bwd_vec_kernel(const uint4* grad_inter, int pitch, const uint4* gate_up, int pitch2, const int* tile_expert, const int* codes,
                   const float* params, const int* total_rows, int nvec, uint4* grad_gate_up, float* row_da,
                   float* row_dg) {
  grid_dep_begin();
  constexpr int RPB = kRowThreads / TPR;
  __shared__ float red[kRowThreads / 32];
  const int total = *total_rows;
  const int t = threadIdx.x % TPR;
  for (long long r0 = static_cast<long long>(blockIdx.x) * RPB; r0 < total; r0 += static_cast<long long>(gridDim.x) * RPB) {
    const long long r = r0 + threadIdx.x / TPR;
    const bool live = r < total;
    const int n = live ? nvec : 0;
    uint4 g[VPT], u[VPT], go[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = t + TPR * i;
      g[i] = c < n ? gate_up[r * pitch2 + c] : make_uint4(0u, 0u, 0u, 0u);
      u[i] = c < n ? gate_up[r * pitch2 + nvec + c] : make_uint4(0u, 0u, 0u, 0u);
      go[i] = c < n ? grad_inter[r * pitch + c] : make_uint4(0u, 0u, 0u, 0u);
    }
    const int e = tile_expert[r0 / B200MOE_TILE_M];
    const int code = codes[e];
    const float alpha = (params != nullptr && code == 5) ? params[2 * e] : 1.0f;
    const float gamma = (params != nullptr && code == 5) ? params[2 * e + 1] : 1.0f;
    uint4* gg = grad_gate_up + r * pitch2;
    uint4* gu = gg + nvec;
    float da = 0.0f, dg = 0.0f;
    switch (code) {                        // uniform over the CTA
      case 1: glu_bwd_row<1, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
      case 2: glu_bwd_row<2, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
      case 5: glu_bwd_row<5, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
      case 6: glu_bwd_row<6, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
      case 7: glu_bwd_row<7, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
      default: glu_bwd_row<0, TPR, VPT>(g, u, go, gg, gu, t, n, alpha, gamma, red, da, dg); break;
    }
    if (row_da != nullptr) {
      if (code == 5) {
        da = row_sum<TPR>(da, red);
        dg = row_sum<TPR>(dg, red);
      }
      if (live && t == 0) {
        row_da[r] = da;
        row_dg[r] = dg;
      }
    }
  }
}

// ---------------------------------------------------------------------------- one value per thread
__global__ void __launch_bounds__(256)
glu_fwd_rows_kernel(const __nv_bfloat16* gate_up, const int* tile_expert, const int* codes, const float* params,
                    const int* total_rows, int I, long long ld2, __nv_bfloat16* inter, long long ldi) {
  grid_dep_begin();
  __shared__ float red[8];
  const int total = *total_rows;
  for (long long r = blockIdx.x; r < total; r += gridDim.x) {
    const int e = tile_expert[r / B200MOE_TILE_M];
    const int code = codes[e];
    const float alpha = (params != nullptr && code == 5) ? params[2 * e] : 1.0f;
    const float gamma = (params != nullptr && code == 5) ? params[2 * e + 1] : 1.0f;
    const __nv_bfloat16* g = gate_up + r * ld2;
    const __nv_bfloat16* u = g + I;
    float inv_r = 1.0f;
    if (is_norm(code)) {
      float ss = 0.0f;
      for (int c = threadIdx.x; c < I; c += blockDim.x) {
        const float v = __bfloat162float(g[c]);
        ss += v * v;
      }
      ss = block_sum(ss, red);
      inv_r = 1.0f / sqrtf(ss / static_cast<float>(I) + kRmsEps);
    }
    for (int c = threadIdx.x; c < I; c += blockDim.x) {
      const float gate = __bfloat162float(g[c]);
      const float up = __bfloat162float(u[c]);
      inter[r * ldi + c] = __float2bfloat16_rn(act_value(code, gate, gate * inv_r, alpha, gamma) * up);
    }
  }
}

// grad_gate_up = [grad_gate | grad_up]; optional per-row d(alpha), d(gamma) for learnable SiTU.
__global__ void __launch_bounds__(256)
glu_bwd_rows_kernel(const __nv_bfloat16* grad_inter, long long ldi, const __nv_bfloat16* gate_up, long long ld2, const int* tile_expert,
                    const int* codes, const float* params, const int* total_rows, int I, __nv_bfloat16* grad_gate_up,
                    float* row_da, float* row_dg) {
  grid_dep_begin();
  __shared__ float red[8];
  const int total = *total_rows;
  for (long long r = blockIdx.x; r < total; r += gridDim.x) {
    const int e = tile_expert[r / B200MOE_TILE_M];
    const int code = codes[e];
    const float alpha = (params != nullptr && code == 5) ? params[2 * e] : 1.0f;
    const float gamma = (params != nullptr && code == 5) ? params[2 * e + 1] : 1.0f;
    const __nv_bfloat16* g = gate_up + r * ld2;
    const __nv_bfloat16* u = g + I;
    const __nv_bfloat16* go = grad_inter + r * ldi;
    __nv_bfloat16* gg = grad_gate_up + r * ld2;
    const bool norm = is_norm(code);
    float rr = 1.0f, S = 0.0f;
    if (norm) {
      float ss = 0.0f;
      for (int c = threadIdx.x; c < I; c += blockDim.x) {
        const float v = __bfloat162float(g[c]);
        ss += v * v;
      }
      ss = block_sum(ss, red);
      rr = sqrtf(ss / static_cast<float>(I) + kRmsEps);
    }
    // derivative of the activation w.r.t. gn, and the activation itself
    auto deriv = [&](float gate, float gn, float& act) -> float {
      const float sig = sigmoidf_(gn);
      if (code == 1 || code == 6) {
        const float rl = fmaxf(gn, 0.0f);
        act = rl * rl;
        return 2.0f * rl;
      }
      if (code == 5) {
        const float t5 = tanh_via_sigmoid(alpha * gate);
        act = gamma * t5 * sig;
        return gamma * (alpha * (1.0f - t5 * t5) * sig + t5 * sig * (1.0f - sig));
      }
      if (code == 7) {
        const float tg = tanh_via_sigmoid(gn);
        act = tg * sig;
        return (1.0f - tg * tg) * sig + tg * sig * (1.0f - sig);
      }
      act = gn * sig;
      return sig * (1.0f + gn * (1.0f - sig));
    };
    if (norm) {   // RMS coupling term S = sum(go * up * f'(gn) * gn)
      float part = 0.0f;
      for (int c = threadIdx.x; c < I; c += blockDim.x) {
        const float gate = __bfloat162float(g[c]);
        const float gn = gate / rr;
        float act;
        const float d = deriv(gate, gn, act);
        part += __bfloat162float(go[c]) * __bfloat162float(u[c]) * d * gn;
      }
      S = block_sum(part, red);
    }
    float da = 0.0f, dg = 0.0f;
    for (int c = threadIdx.x; c < I; c += blockDim.x) {
      const float gate = __bfloat162float(g[c]);
      const float up = __bfloat162float(u[c]);
      const float gi = __bfloat162float(go[c]);
      const float gn = norm ? gate / rr : gate;
      float act;
      const float d = deriv(gate, gn, act);
      const float gu_ = gi * up;
      const float grad_gate = norm ? (gu_ * d - (S / static_cast<float>(I)) * gn) / rr : gu_ * d;
      gg[c] = __float2bfloat16_rn(grad_gate);
      gg[I + c] = __float2bfloat16_rn(gi * act);
      if (row_da != nullptr && code == 5) {
        const float sig = sigmoidf_(gate);
        const float t5 = tanh_via_sigmoid(alpha * gate);
        da += gu_ * gamma * gate * (1.0f - t5 * t5) * sig;
        dg += gu_ * t5 * sig;
      }
    }
    if (row_da != nullptr) {
      da = block_sum(da, red);
      dg = block_sum(dg, red);
      if (threadIdx.x == 0) {
        row_da[r] = da;
        row_dg[r] = dg;
      }
    }
  }
}

// out[e] = (sum of row_da over the rows of e, sum of row_dg): deterministic, one CTA per expert.  Bound by the latency
// of its loads: 1024 threads keep a segment's rows in flight in a few rounds (3000 rows an expert: 8.7 -> 4.1 us with 256 -> 1024).
constexpr int kSumThreads = 1024;
__global__ void __launch_bounds__(kSumThreads)
expert_row_sums_kernel(const float* row_da, const float* row_dg, const int* poffs, float* out) {
  grid_dep_begin();
  __shared__ float red[kSumThreads / 32];
  const int e = blockIdx.x;
  float a = 0.0f, b = 0.0f;
  for (int r = poffs[e] + threadIdx.x; r < poffs[e + 1]; r += blockDim.x) {
    a += row_da[r];
    b += row_dg[r];
  }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) {
    out[2 * e] = a;
    out[2 * e + 1] = b;
  }
}

// rows of the special experts (those after the first `first_special` experts):
// dst[r] = src[r] for Identity (code 3), 0 otherwise (Zero, code 4); TPR threads share a row
template <int TPR>
__global__ void __launch_bounds__(256)
special_rows_kernel(const uint4* src, const int* tile_expert, const int* codes, const int* poffs, int first_special,
                    int num_experts, int vec_per_row, int pitch_src, int pitch, uint4* dst) {
  grid_dep_begin();
  constexpr int G = 256 / TPR;
  const int r0 = poffs[first_special], r1 = poffs[num_experts];
  for (long long r = r0 + static_cast<long long>(blockIdx.x) * G + threadIdx.x / TPR; r < r1;
       r += static_cast<long long>(gridDim.x) * G) {
    const bool copy = codes[tile_expert[r / B200MOE_TILE_M]] == 3;
    for (int c = threadIdx.x % TPR; c < vec_per_row; c += TPR)
      dst[r * pitch + c] = copy ? src[r * pitch_src + c] : make_uint4(0u, 0u, 0u, 0u);
  }
}

static long long ceil_div64(long long a, long long b) { return (a + b - 1) / b; }
static int rows_grid(long long rows_cap) {
  long long g = rows_cap;
  const long long cap = static_cast<long long>(num_sms()) * 16;
  if (g > cap) g = cap;
  return static_cast<int>(g < 1 ? 1 : g);
}

// The register-resident kernels take 16-byte-aligned rows of at most 8192 values
constexpr int64_t kMaxVecWidth = 8192;
static bool rows_in_registers(int64_t I, const void* a, const void* b, const void* c) {
  return I % 8 == 0 && I <= kMaxVecWidth && aligned16(a) && aligned16(b) && aligned16(c);
}
// f(TPR, VPT): the narrowest row group that holds nvec vectors, of two or three vectors of each operand a thread: from d_ff 344 on at most
// a third of its lanes is idle (d_ff 768: 32 x 3, 1032: 64 x 3; d_ff 256 uses half of 32 x 2); beside more registers, fewer warps a row need
// fewer barriers
template <class F>
static void by_row_width(int nvec, F f) {
  auto width = [&](auto tpr) {
    if (nvec <= 2 * tpr.value) f(tpr, std::integral_constant<int, 2>());
    else f(tpr, std::integral_constant<int, 3>());
  };
  if (nvec <= 96) width(std::integral_constant<int, 32>());
  else if (nvec <= 192) width(std::integral_constant<int, 64>());
  else if (nvec <= 384) width(std::integral_constant<int, 128>());
  else if (nvec <= 768) width(std::integral_constant<int, 256>());
  else f(std::integral_constant<int, 256>(), std::integral_constant<int, 4>());
}

int glu_fwd_rows(const void* gate_up, int64_t ld2, const int32_t* tile_expert, const int32_t* act_codes, const float* act_params,
                 const int32_t* total_rows, int64_t rows_cap, int64_t I, void* inter, int64_t ldi, b200moe_stream_t stream) {
  B200_CHECK_ARG(gate_up && tile_expert && act_codes && total_rows && inter, B200MOE_E_NULL, "glu_fwd_rows: null pointer");
  B200_CHECK_ARG(I > 0, B200MOE_E_BAD_SHAPE, "glu_fwd_rows: I = %lld", (long long)I);
  if (rows_cap <= 0) return 0;
  if (rows_in_registers(I, gate_up, inter, inter)) {
    const int nvec = static_cast<int>(I / 8);
    cudaError_t err = cudaSuccess;
    by_row_width(nvec, [&](auto tpr, auto vpt) {
      err = launch_chained(glu_fwd_vec_kernel<tpr.value, vpt.value>, rows_grid(ceil_div64(rows_cap, kRowThreads / tpr.value)),
                           kRowThreads, 0, (cudaStream_t)stream, 1, reinterpret_cast<const uint4*>(gate_up), tile_expert, act_codes,
                           act_params, total_rows, nvec, static_cast<int>(ld2 / 8), reinterpret_cast<uint4*>(inter), static_cast<int>(ldi / 8));
    });
    B200_CUDA(err);
    return 0;
  }
  B200_LAUNCH(glu_fwd_rows_kernel, rows_grid(rows_cap), 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(gate_up), tile_expert,
              act_codes, act_params, total_rows, static_cast<int>(I), static_cast<long long>(ld2), reinterpret_cast<__nv_bfloat16*>(inter),
              static_cast<long long>(ldi));
  return 0;
}

int glu_bwd_rows(const void* grad_inter, int64_t ldi, const void* gate_up, int64_t ld2, const int32_t* tile_expert, const int32_t* act_codes,
                 const float* act_params, const int32_t* total_rows, int64_t rows_cap, int64_t I, void* grad_gate_up, float* row_da, float* row_dg,
                 b200moe_stream_t stream) {
  B200_CHECK_ARG(grad_inter && gate_up && tile_expert && act_codes && total_rows && grad_gate_up, B200MOE_E_NULL,
                 "glu_bwd_rows: null pointer");
  B200_CHECK_ARG((row_da == nullptr) == (row_dg == nullptr), B200MOE_E_NULL, "glu_bwd_rows: row_da and row_dg go together");
  B200_CHECK_ARG(I > 0, B200MOE_E_BAD_SHAPE, "glu_bwd_rows: I = %lld", (long long)I);
  if (rows_cap <= 0) return 0;
  if (rows_in_registers(I, grad_inter, gate_up, grad_gate_up)) {
    const int nvec = static_cast<int>(I / 8);
    cudaError_t err = cudaSuccess;
    by_row_width(nvec, [&](auto tpr, auto vpt) {
      err = launch_chained(glu_bwd_vec_kernel<tpr.value, vpt.value>, rows_grid(ceil_div64(rows_cap, kRowThreads / tpr.value)),
                           kRowThreads, 0, (cudaStream_t)stream, 1, reinterpret_cast<const uint4*>(grad_inter),
                           static_cast<int>(ldi / 8), reinterpret_cast<const uint4*>(gate_up), static_cast<int>(ld2 / 8), tile_expert, act_codes, act_params, total_rows, nvec,
                           reinterpret_cast<uint4*>(grad_gate_up), row_da, row_dg);
    });
    B200_CUDA(err);
    return 0;
  }
  B200_LAUNCH(glu_bwd_rows_kernel, rows_grid(rows_cap), 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(grad_inter),
              static_cast<long long>(ldi), reinterpret_cast<const __nv_bfloat16*>(gate_up), static_cast<long long>(ld2), tile_expert, act_codes, act_params, total_rows, static_cast<int>(I),
              reinterpret_cast<__nv_bfloat16*>(grad_gate_up), row_da, row_dg);
  return 0;
}

int special_rows(const void* src, int64_t lds, const int32_t* tile_expert, const int32_t* act_codes, const int32_t* poffs, int first_special,
                 int num_experts, int64_t H, int64_t ldh, int64_t rows_cap, void* dst, b200moe_stream_t stream) {
  B200_CHECK_ARG(src && tile_expert && act_codes && poffs && dst, B200MOE_E_NULL, "special_rows: null pointer");
  B200_CHECK_ARG(H > 0 && H % 8 == 0 && first_special >= 0 && first_special <= num_experts, B200MOE_E_BAD_SHAPE,
                 "special_rows: H = %lld, first_special = %d, num_experts = %d", (long long)H, first_special, num_experts);
  B200_CHECK_ARG(aligned16(src) && aligned16(dst), B200MOE_E_ALIGN, "special_rows: pointers must be 16-byte aligned");
  if (rows_cap <= 0 || first_special == num_experts) return 0;
  cudaError_t err = cudaSuccess;
  by_row_threads(static_cast<int>(H / 8), [&](auto tpr) {
    err = launch_chained(special_rows_kernel<tpr.value>, rows_grid(ceil_div64(rows_cap, 256 / tpr.value)), 256, 0,
                         (cudaStream_t)stream, 1, reinterpret_cast<const uint4*>(src), tile_expert, act_codes, poffs,
                         first_special, num_experts, static_cast<int>(H / 8), static_cast<int>(lds / 8), static_cast<int>(ldh / 8), reinterpret_cast<uint4*>(dst));
  });
  B200_CUDA(err);
  return 0;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_glu_fwd_rows(const void* gate_up, const int32_t* tile_expert, const int32_t* act_codes,
                         const float* act_params, const int32_t* total_rows, int64_t rows_cap, int64_t I, void* inter,
                         b200moe_stream_t stream) {
  return glu_fwd_rows(gate_up, 2 * I, tile_expert, act_codes, act_params, total_rows, rows_cap, I, inter, I, stream);
}

int b200moe_glu_bwd_rows(const void* grad_inter, const void* gate_up, const int32_t* tile_expert,
                         const int32_t* act_codes, const float* act_params, const int32_t* total_rows, int64_t rows_cap,
                         int64_t I, void* grad_gate_up, float* row_da, float* row_dg, b200moe_stream_t stream) {
  return glu_bwd_rows(grad_inter, I, gate_up, 2 * I, tile_expert, act_codes, act_params, total_rows, rows_cap, I, grad_gate_up, row_da, row_dg, stream);
}

int b200moe_expert_row_sums(const float* row_da, const float* row_dg, const int32_t* poffs, int E, float* out,
                            b200moe_stream_t stream) {
  B200_CHECK_ARG(row_da && row_dg && poffs && out, B200MOE_E_NULL, "expert_row_sums: null pointer");
  B200_CHECK_ARG(E >= 1, B200MOE_E_BAD_SHAPE, "expert_row_sums: E = %d", E);
  B200_LAUNCH(expert_row_sums_kernel, E, kSumThreads, 0, stream, row_da, row_dg, poffs, out);
  return 0;
}

int b200moe_special_rows(const void* src, const int32_t* tile_expert, const int32_t* act_codes, const int32_t* poffs,
                         int first_special, int num_experts, int64_t H, int64_t rows_cap, void* dst,
                         b200moe_stream_t stream) {
  return special_rows(src, H, tile_expert, act_codes, poffs, first_special, num_experts, H, H, rows_cap, dst, stream);
}

}  // extern "C"
