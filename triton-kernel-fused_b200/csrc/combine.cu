// Weighted combine (forward), its backward, both as gather-reduce passes over 16-byte vectors.
// Deterministic: every output element is produced by exactly one thread, no atomics.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace b200moe {

__device__ __forceinline__ void fma8(float (&acc)[8], const uint4& v, float w) {
  const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  acc[0] += w * a.x; acc[1] += w * a.y; acc[2] += w * b.x; acc[3] += w * b.y;
  acc[4] += w * c.x; acc[5] += w * c.y; acc[6] += w * d.x; acc[7] += w * d.y;
}

constexpr int kVecBatch = 4;   // 16-byte vectors a lane keeps in flight per row it reads

// out[t] = sum_j w[t,j] * rows[slot_row[t*k+j]] (+ add[t])  (fp32 accumulate in slot order j = 0..k-1).  `add` is the
// router's share of grad_x: adding it here saves the pass of a separate addition (headline layer: 32 us).
// Bound: HBM, k rows in and one out a token.  TPR threads share a token, so that a narrow row does not leave most of a CTA
// idle; a thread reads its token's table entries itself (a broadcast) and keeps four rows' vectors in flight.
// Against one CTA of 256 threads a token: 20 000 tokens of H 256, top-8 80 -> 29 us, 16 384 of H 512, top-2 21 -> 12 us, 32 768 of
// H 2048, top-8 223 -> 214 us.
// PITCH: rows lie further apart than they are long.  As a launch parameter alone it made the rest slower: 4096 tokens of H 1024
// 6.2 -> 6.5 us, 8192 of H 512 6.1 -> 6.6; with a kernel of each kind 6.2 and 6.1.
template <int TPR, bool PITCH>
__global__ void __launch_bounds__(256)
combine_kernel(const uint4* rows, int pitch, const float* w, const int* slot_row, const uint4* add, long long T, int k,
               int vec_per_row, uint4* out) {
  grid_dep_begin();
  constexpr int G = 256 / TPR;
  for (long long t = static_cast<long long>(blockIdx.x) * G + threadIdx.x / TPR; t < T;
       t += static_cast<long long>(gridDim.x) * G) {
    const int* slots = slot_row + t * k;
    for (int c = threadIdx.x % TPR; c < vec_per_row; c += TPR) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j0 = 0; j0 < k; j0 += 4) {
        int r[4];
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = j0 + i < k ? slots[j0 + i] : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i)   // a slot without a row (its expert index was out of range) adds nothing
          if (r[i] >= 0) v[i] = rows[static_cast<long long>(r[i]) * (PITCH ? pitch : vec_per_row) + c];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (r[i] >= 0) fma8(acc, v[i], w != nullptr ? w[t * k + j0 + i] : 1.0f);
      }
      if (add != nullptr) fma8(acc, add[t * vec_per_row + c], 1.0f);
      uint4 o;
      o.x = pack_bf16x2(acc[0], acc[1]);
      o.y = pack_bf16x2(acc[2], acc[3]);
      o.z = pack_bf16x2(acc[4], acc[5]);
      o.w = pack_bf16x2(acc[6], acc[7]);
      out[t * vec_per_row + c] = o;
    }
  }
}

// grad_eo[r] = bf16(go[tok] * w[slot]);  grad_w[slot] = sum_h go[tok,h] * eo[r,h]  (fp32)
// One warp per routed row, 2 * kVecBatch independent 16-byte loads in flight per lane; the dot product is
// reduced by shuffles in a fixed order.
__global__ void __launch_bounds__(256)
combine_bwd_kernel(const uint4* go, const uint4* eo, const float* w, const int* row_slot, const int* total_rows, int k,
                   int vec_per_row, int pitch, uint4* grad_eo, float* grad_w) {
  grid_dep_begin();
  const int lane = threadIdx.x & 31;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const int total = *total_rows;
  for (long long r = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < total; r += warps) {
    const int slot = row_slot[r];
    uint4* dst = grad_eo + r * pitch;
    if (slot < 0) {
      for (int c = lane; c < vec_per_row; c += 32) dst[c] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const float wt = w[slot];
    const uint4* g = go + static_cast<long long>(slot / k) * vec_per_row;
    const uint4* e = eo + r * pitch;
    float dot = 0.0f;
    for (int c0 = 0; c0 < vec_per_row; c0 += 32 * kVecBatch) {
      uint4 gv[kVecBatch], ev[kVecBatch];
#pragma unroll
      for (int i = 0; i < kVecBatch; ++i) {
        const int c = c0 + 32 * i + lane;
        gv[i] = c < vec_per_row ? g[c] : make_uint4(0u, 0u, 0u, 0u);
        ev[i] = c < vec_per_row ? e[c] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int i = 0; i < kVecBatch; ++i) {
        const int c = c0 + 32 * i + lane;
        const float2 g0 = unpack_bf16x2(gv[i].x), g1 = unpack_bf16x2(gv[i].y), g2 = unpack_bf16x2(gv[i].z),
                     g3 = unpack_bf16x2(gv[i].w);
        const float2 e0 = unpack_bf16x2(ev[i].x), e1 = unpack_bf16x2(ev[i].y), e2 = unpack_bf16x2(ev[i].z),
                     e3 = unpack_bf16x2(ev[i].w);
        dot += g0.x * e0.x + g0.y * e0.y + g1.x * e1.x + g1.y * e1.y + g2.x * e2.x + g2.y * e2.y + g3.x * e3.x +
               g3.y * e3.y;
        if (c < vec_per_row) {
          uint4 o;
          o.x = pack_bf16x2(g0.x * wt, g0.y * wt);
          o.y = pack_bf16x2(g1.x * wt, g1.y * wt);
          o.z = pack_bf16x2(g2.x * wt, g2.y * wt);
          o.w = pack_bf16x2(g3.x * wt, g3.y * wt);
          dst[c] = o;
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
    if (lane == 0) grad_w[slot] = dot;
  }
}

// The same for rows of at most 32 vectors: a lane has one vector of each of four rows, so that a warp keeps eight loads a lane
// in flight here too (the kernel above keeps two: 20 000 tokens of H 256, top-8: 82 -> 70 us; for wider rows it is the
// faster one: 64 vectors 18 against 24 us, 256 vectors 200 against 248 us).
__global__ void __launch_bounds__(256)
combine_bwd_narrow_kernel(const uint4* go, const uint4* eo, const float* w, const int* row_slot, const int* total_rows,
                          int k, int vec_per_row, int pitch, uint4* grad_eo, float* grad_w) {
  grid_dep_begin();
  constexpr int RB = 4;
  const int lane = threadIdx.x & 31;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const int total = *total_rows;
  const bool in = lane < vec_per_row;
  for (long long r0 = ((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * RB; r0 < total; r0 += warps * RB) {
    int slot[RB];
    float wt[RB];
    uint4 g[RB], e[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) slot[q] = r0 + q < total ? row_slot[r0 + q] : -1;
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const bool live = in && slot[q] >= 0;
      wt[q] = slot[q] >= 0 ? w[slot[q]] : 0.0f;
      g[q] = live ? go[static_cast<long long>(slot[q] / k) * vec_per_row + lane] : make_uint4(0u, 0u, 0u, 0u);
      e[q] = live ? eo[(r0 + q) * pitch + lane] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const uint32_t gw[4] = {g[q].x, g[q].y, g[q].z, g[q].w}, ew[4] = {e[q].x, e[q].y, e[q].z, e[q].w};
      uint32_t o[4];
      float dot = 0.0f;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float2 gf = unpack_bf16x2(gw[h]), ef = unpack_bf16x2(ew[h]);
        dot += gf.x * ef.x + gf.y * ef.y;
        o[h] = slot[q] >= 0 ? pack_bf16x2(gf.x * wt[q], gf.y * wt[q]) : 0u;
      }
      if (in && r0 + q < total) grad_eo[(r0 + q) * pitch + lane] = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
      if (lane == 0 && slot[q] >= 0) grad_w[slot[q]] = dot;
    }
  }
}

int combine_add(const void* rows, int64_t ldh, const float* w, const int32_t* slot_row, const void* add, int64_t T, int k, int64_t H, void* out,
                b200moe_stream_t stream) {
  B200_CHECK_ARG(rows && slot_row && out, B200MOE_E_NULL, "combine: null pointer");
  B200_CHECK_ARG(H > 0 && H % 8 == 0, B200MOE_E_BAD_SHAPE, "combine: H = %lld must be a multiple of 8", (long long)H);
  B200_CHECK_ARG(k >= 1 && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE, "combine: k = %d", k);
  B200_CHECK_ARG(aligned16(rows) && aligned16(out) && aligned16(add), B200MOE_E_ALIGN, "combine: pointers must be 16-byte aligned");
  if (T <= 0) return 0;
  cudaError_t err = cudaSuccess;
  by_row_threads(static_cast<int>(H / 8), [&](auto tpr) {
    constexpr int G = 256 / tpr.value;
    const long long grid = std::min<long long>((T + G - 1) / G, static_cast<long long>(num_sms()) * 16);
    err = launch_chained(ldh != H ? combine_kernel<tpr.value, true> : combine_kernel<tpr.value, false>, static_cast<int>(grid), 256, 0,
                         (cudaStream_t)stream, 1,
                         reinterpret_cast<const uint4*>(rows), static_cast<int>(ldh / 8), w, slot_row, reinterpret_cast<const uint4*>(add), T, k,
                         static_cast<int>(H / 8), reinterpret_cast<uint4*>(out));
  });
  B200_CUDA(err);
  return 0;
}

int combine_bwd(const void* grad_out, const void* eo, const float* w, const int32_t* row_slot, const int32_t* total_rows, int k, int64_t H,
                int64_t ldh, int64_t rows_cap, void* grad_eo, float* grad_w, b200moe_stream_t stream) {
  B200_CHECK_ARG(grad_out && eo && w && row_slot && total_rows && grad_eo && grad_w, B200MOE_E_NULL,
                 "combine_bwd: null pointer");
  B200_CHECK_ARG(H > 0 && H % 8 == 0, B200MOE_E_BAD_SHAPE, "combine_bwd: H = %lld must be a multiple of 8", (long long)H);
  B200_CHECK_ARG(k >= 1, B200MOE_E_BAD_SHAPE, "combine_bwd: k = %d", k);
  B200_CHECK_ARG(aligned16(grad_out) && aligned16(eo) && aligned16(grad_eo), B200MOE_E_ALIGN,
                 "combine_bwd: pointers must be 16-byte aligned");
  if (rows_cap <= 0) return 0;
  const int nvec = static_cast<int>(H / 8), rows_per_warp = nvec <= 32 ? 4 : 1;
  const long long grid = std::min<long long>((rows_cap + 8 * rows_per_warp - 1) / (8 * rows_per_warp), static_cast<long long>(num_sms()) * 8);
  auto kernel = nvec <= 32 ? combine_bwd_narrow_kernel : combine_bwd_kernel;
  B200_LAUNCH(kernel, static_cast<int>(grid), 256, 0, stream, reinterpret_cast<const uint4*>(grad_out),
              reinterpret_cast<const uint4*>(eo), w, row_slot, total_rows, k, nvec, static_cast<int>(ldh / 8), reinterpret_cast<uint4*>(grad_eo), grad_w);
  return 0;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_combine(const void* rows, const float* w, const int32_t* slot_row, int64_t T, int k, int64_t H,
                    void* out, b200moe_stream_t stream) {
  return combine_add(rows, H, w, slot_row, nullptr, T, k, H, out, stream);
}

int b200moe_combine_add(const void* rows, const float* w, const int32_t* slot_row, const void* add, int64_t T, int k,
                        int64_t H, void* out, b200moe_stream_t stream) {
  return combine_add(rows, H, w, slot_row, add, T, k, H, out, stream);
}

int b200moe_combine_bwd(const void* grad_out, const void* eo, const float* w, const int32_t* row_slot,
                        const int32_t* total_rows, int k, int64_t H, int64_t rows_cap, void* grad_eo, float* grad_w,
                        b200moe_stream_t stream) {
  return combine_bwd(grad_out, eo, w, row_slot, total_rows, k, H, H, rows_cap, grad_eo, grad_w, stream);
}

}  // extern "C"
