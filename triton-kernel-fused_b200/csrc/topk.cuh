// Top-k of a token's experts inside one warp: shared by the router epilogue kernels and the small batch's router GEMM.
// Lane l holds experts l, l+32, ... (VPL values).
#pragma once
#include <type_traits>

#include "common.cuh"

namespace b200moe {

constexpr int kMaxVpl = B200MOE_MAX_EXPERTS / 32;  // most values a lane holds

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// A selection value as an unsigned key of the same order (+0 and -0 alike; NaN above infinity).  Key 0 lies below
// every value: experts that do not exist.  A picked expert falls to the key of -1e30, as in the reference.
__device__ __forceinline__ uint32_t select_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr uint32_t kKnockOut = ~0xf149f2cau;   // select_key(-1e30f)

// The k picks of the token whose scores and selection keys a warp holds: lane j < k gets pick j and its weight.
template <int VPL>
__device__ __forceinline__ void topk_of_token(const float (&sc)[VPL], uint32_t (&key)[VPL], int k, int norm, float scale,
                                              int* hist, bool count, int& my_idx, float& my_w) {
  const int lane = threadIdx.x & 31;
  my_idx = 0;
  my_w = 0.0f;
  for (int j = 0; j < k; ++j) {
    // lane-local best: ascending i = ascending expert id, strict '>' keeps the lowest id
    uint32_t bk = key[0];
    int bi = lane;
#pragma unroll
    for (int i = 1; i < VPL; ++i) {
      if (key[i] > bk) {
        bk = key[i];
        bi = lane + 32 * i;
      }
    }
    const uint32_t best = __reduce_max_sync(0xffffffffu, bk);
    bi = static_cast<int>(__reduce_min_sync(0xffffffffu, bk == best ? static_cast<unsigned>(bi) : 0xffffffffu));
    // owner lane hands out the unbiased score and knocks the pick out
    float wv = 0.0f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (bi == lane + 32 * i) {
        wv = sc[i];
        key[i] = kKnockOut;
      }
    }
    wv = __shfl_sync(0xffffffffu, wv, bi & 31);
    if (lane == j) {
      my_idx = bi;
      my_w = wv;
    }
  }
  if (count && lane < k) atomicAdd(&hist[my_idx], 1);
  if (norm && k > 1) {
    float tsum = 0.0f;
    for (int j = 0; j < k; ++j) tsum += __shfl_sync(0xffffffffu, my_w, j);  // fixed order
    tsum += 1e-20f;
    my_w = my_w / tsum;
  }
  my_w = my_w * scale;
}

// f(VPL) for E experts
template <class F>
static void by_experts(int E, F f) {
  if (E <= 32) f(std::integral_constant<int, 1>());
  else if (E <= 64) f(std::integral_constant<int, 2>());
  else if (E <= 128) f(std::integral_constant<int, 4>());
  else f(std::integral_constant<int, kMaxVpl>());
}

}  // namespace b200moe
