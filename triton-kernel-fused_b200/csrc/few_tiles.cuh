// Tiles of the grouped products for few rows per expert (gemm_few.cu, gemm_mxfp8.cu): (expert, chunk of its rows, block of
// output columns), found on the device from the experts' row counts; and the way a result leaves such a tile's accumulator.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace b200moe {

struct FewTile { int e, m0, row0, live; };

// pre[e] = chunks of at most NT rows in front of expert e, pre[B200MOE_MAX_EXPERTS] all of them: one warp, a lane takes 8
// neighbouring experts.  The counts are read from L2: before the wait for an earlier kernel an L1 line may be older than the launch.
template <int NT>
__device__ __forceinline__ void few_prefix(const int* counts, int E, int lane, int* pre) {
  constexpr int V = B200MOE_MAX_EXPERTS / 32;
  int c[V], sum = 0;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int e = lane * V + i;
    c[i] = e < E ? (__ldcg(counts + e) + NT - 1) / NT : 0;
    sum += c[i];
  }
  int incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += o;
  }
  int run = incl - sum;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    pre[lane * V + i] = run;
    run += c[i];
  }
  if (lane == 31) pre[B200MOE_MAX_EXPERTS] = run;
}

// The tile of an index: N output columns in blocks of TM, the rows of expert e from first_row[e] on.  before_wait: as above
template <int NT, int TM>
__device__ __forceinline__ FewTile few_tile(const int* counts, const int* first_row, int E, int N, const int* pre, int tile,
                                            bool before_wait = false) {
  const int mt = (N + TM - 1) / TM;
  const int c = tile / mt;
  int lo = 0, hi = E;                         // the last expert with pre[e] <= c
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pre[mid] <= c) lo = mid;
    else hi = mid;
  }
  FewTile t;
  t.e = lo;
  t.m0 = (tile - c * mt) * TM;
  const int first = (c - pre[lo]) * NT;
  t.row0 = (before_wait ? __ldcg(first_row + lo) : first_row[lo]) + first;
  t.live = min(NT, (before_wait ? __ldcg(counts + lo) : counts[lo]) - first);
  return t;
}

// 16 accumulator columns (rows of X) of a warp's 32 lanes (output columns), rounded to bf16: v[h][2b + i] = rows 8b + 2 (lane % 4) and the
// next one of column lane / 4 of the block 2h + i of 8 output columns
__device__ __forceinline__ void few_fetch(uint32_t taddr, uint32_t (&v)[2][4]) {
  uint32_t r[2][8];
  tmem_ld_blocks16(taddr, r[0]);
  tmem_ld_blocks16(taddr + (16u << 16), r[1]);
  tmem_ld_wait();
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) v[h][i] = pack_bf16x2(__uint_as_float(r[h][2 * i]), __uint_as_float(r[h][2 * i + 1]));
}
// ... turned: w = the 8 output columns of block lane % 4 for row 8b + lane / 4
__device__ __forceinline__ void few_turn(const uint32_t (&v)[2][4], int b, int lane, uint32_t (&w)[4]) {
  w[0] = movmatrix_trans(v[0][2 * b]);
  w[1] = movmatrix_trans(v[0][2 * b + 1]);
  w[2] = movmatrix_trans(v[1][2 * b]);
  w[3] = movmatrix_trans(v[1][2 * b + 1]);
  quad_transpose(w, lane);
}

}  // namespace b200moe
