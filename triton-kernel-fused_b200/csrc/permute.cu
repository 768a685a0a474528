// Expert permutation as a stable counting sort on the device (no host sync).  A CTA owns a run of consecutive slots, a
// warp a run of 32 * PL of them:
//   1. hist : (only when the slots fill more than one CTA) per-expert histogram of every CTA's run
//   2. rank : every warp walks its run once (__match_any_sync groups equal experts) and keeps each slot's rank inside
//             the run; a prefix over the CTA's warps, the earlier CTAs' histograms and the experts then gives
//             compact and padded offsets, tile table, pad-row markers -> slot_row / row_slot / order
// Row r of expert e is therefore the r-th smallest slot index t*k+j with idx[t,j] == e, which is
// exactly what a stable sort of idx.flatten() gives.
//
// Bound: launch and load latency, not bytes (98 304 slots are 0.8 MB).  Every load of a thread is issued before its
// first use, every CTA derives the offsets it needs by itself (a row of E counts per CTA to add up) instead
// of waiting for a one-CTA scan between the passes, and up to 1024 slots take one launch.
// Against one warp per 512 slots with a serial scan between: 98 304 slots over 64 experts 35.5 -> 7.6 us, 262 144 over
// 128 67 -> 10.9 us, 288 over 64 23.9 -> 4.3 us.
#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace b200moe {

constexpr int kMaxVals = B200MOE_MAX_EXPERTS / 32;   // experts a lane holds in the scan over the experts

// How the slots are dealt out: warps per CTA and slots per lane.  A warp's walk costs a __match_any_sync per 32 slots,
// whose time grows with the distinct experts among them, so a large sort wants its walks on many SMs; but every CTA
// adds up one histogram row per CTA, so the runs grow with the number of slots.  4000 slots over 64 experts: one CTA of 32
// warps 9.7 us, four CTAs of 8 warps 4.5 + 1.8 us (with the histogram launch); 9000 slots: one CTA 20 us, nine 4.5 + 1.8 us.
struct PermSplit { int warps, per_lane; };
static PermSplit perm_split(long long M) {
  if (M <= (1LL << 17)) return {8, 4};      // up to 1024 slots: one CTA, one launch
  if (M <= (1LL << 18)) return {16, 4};
  if (M <= (1LL << 20)) return {32, 4};
  return {32, 16};
}

template <int W, int PL>
__global__ void __launch_bounds__(32 * W)
permute_hist_kernel(const long long* idx, long long M, int E, int* block_hist) {
  grid_dep_begin();
  constexpr int kPermThreads = 32 * W;
  __shared__ int h[B200MOE_MAX_EXPERTS];
  for (int e = threadIdx.x; e < E; e += kPermThreads) h[e] = 0;
  const long long s0 = static_cast<long long>(blockIdx.x) * (PL * kPermThreads) + threadIdx.x;
  long long v[PL];
#pragma unroll
  for (int i = 0; i < PL; ++i) v[i] = s0 + i * kPermThreads < M ? idx[s0 + i * kPermThreads] : -1;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PL; ++i)
    if (v[i] >= 0 && v[i] < E) atomicAdd(&h[v[i]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kPermThreads) block_hist[static_cast<long long>(blockIdx.x) * E + e] = h[e];
}

template <int W, int PL>
__global__ void __launch_bounds__(32 * W)
permute_rank_kernel(const long long* idx, long long M, int E, const int* block_hist, int* counts, int* offs, int* poffs,
                    int* slot_row, int* row_slot, int* tile_expert, int* order, int* slot_pos, int* counts_out,
                    long long* load, int* status) {
  grid_dep_begin();
  constexpr int kPermWarps = W, kPermThreads = 32 * W;
  extern __shared__ int sh[];                          // [W][E]: ranks a warp's run starts at
  __shared__ int s_before[B200MOE_MAX_EXPERTS];        // slots of the expert in earlier CTAs
  __shared__ int s_cnt[B200MOE_MAX_EXPERTS];           // ... in all CTAs
  __shared__ int s_off[B200MOE_MAX_EXPERTS + 1], s_poff[B200MOE_MAX_EXPERTS + 1];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  int* wh = sh + warp * E;
  const long long s0 = (static_cast<long long>(blockIdx.x) * kPermWarps + warp) * (PL * 32) + lane;
  int ex[PL], rank[PL];
  {
    long long v[PL];
#pragma unroll
    for (int i = 0; i < PL; ++i) v[i] = s0 + 32 * i < M ? idx[s0 + 32 * i] : -1;
    for (int e = lane; e < E; e += 32) wh[e] = 0;
    for (int e = threadIdx.x; e < E; e += kPermThreads) s_before[e] = s_cnt[e] = 0;
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      ex[i] = (v[i] >= 0 && v[i] < E) ? static_cast<int>(v[i]) : -1;
      if (ex[i] < 0 && s0 + 32 * i < M) atomicCAS(status, 0, ST_BAD_EXPERT_INDEX);
    }
  }
  __syncthreads();
  // counts of the other CTAs: the threads split the rows, E at a time
  if (gridDim.x > 1) {
    const int rows_at_once = kPermThreads / E;         // at least 1: 256 threads, 256 experts
    const int e = threadIdx.x % E, r0 = threadIdx.x / E;
    if (r0 < rows_at_once) {
      int before = 0, all = 0;
      for (int r = r0; r < static_cast<int>(gridDim.x); r += 8 * rows_at_once) {
        int c[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = r + i * rows_at_once;
          c[i] = rr < static_cast<int>(gridDim.x) ? block_hist[static_cast<long long>(rr) * E + e] : 0;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          all += c[i];
          before += (r + i * rows_at_once < static_cast<int>(blockIdx.x)) ? c[i] : 0;
        }
      }
      if (before != 0) atomicAdd(&s_before[e], before);
      if (all != 0) atomicAdd(&s_cnt[e], all);
    }
  }
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const unsigned peers = __match_any_sync(0xffffffffu, ex[i]);
    const unsigned lower = peers & ((1u << lane) - 1);
    rank[i] = ex[i] >= 0 ? wh[ex[i]] + __popc(lower) : 0;
    __syncwarp();
    if (ex[i] >= 0 && lower == 0) wh[ex[i]] += __popc(peers);   // group leader
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < E) {          // ranks at which every warp's run starts
    const int e = threadIdx.x;
    int run = s_before[e];
#pragma unroll
    for (int w = 0; w < kPermWarps; ++w) {
      const int c = sh[w * E + e];
      sh[w * E + e] = run;
      run += c;
    }
    if (gridDim.x == 1) s_cnt[e] = run;
  }
  __syncthreads();
  if (warp == 0) {                // offsets of the experts: a lane takes kMaxVals neighbours, then a scan over the lanes
    int c[kMaxVals], a = 0, b = 0;
#pragma unroll
    for (int i = 0; i < kMaxVals; ++i) {
      const int e = lane * kMaxVals + i;
      c[i] = e < E ? s_cnt[e] : 0;
      a += c[i];
      b += (c[i] + B200MOE_TILE_M - 1) / B200MOE_TILE_M * B200MOE_TILE_M;
    }
    int ia = a, ib = b;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int pa = __shfl_up_sync(0xffffffffu, ia, off), pb = __shfl_up_sync(0xffffffffu, ib, off);
      if (lane >= off) {
        ia += pa;
        ib += pb;
      }
    }
    a = ia - a;
    b = ib - b;
#pragma unroll
    for (int i = 0; i < kMaxVals; ++i) {
      const int e = lane * kMaxVals + i;
      if (e <= E) {
        s_off[e] = a;
        s_poff[e] = b;
      }
      a += c[i];
      b += (c[i] + B200MOE_TILE_M - 1) / B200MOE_TILE_M * B200MOE_TILE_M;
    }
    if (lane == 31 && E == B200MOE_MAX_EXPERTS) {
      s_off[E] = a;
      s_poff[E] = b;
    }
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e <= E; e += kPermThreads) {
      offs[e] = s_off[e];
      poffs[e] = s_poff[e];
      if (e == E) continue;
      counts[e] = s_cnt[e];
      if (counts_out != nullptr) counts_out[e] = s_cnt[e];
      if (load != nullptr) load[e] += s_cnt[e];
    }
  for (int e = blockIdx.x * kPermWarps + warp; e < E; e += gridDim.x * kPermWarps) {
    const int p0 = s_poff[e], p1 = s_poff[e + 1];
    for (int r = p0 + s_cnt[e] + lane; r < p1; r += 32) row_slot[r] = -1;          // pad rows of this expert
    for (int t = p0 / B200MOE_TILE_M + lane; t < p1 / B200MOE_TILE_M; t += 32) tile_expert[t] = e;
  }
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const long long s = s0 + 32 * i;
    if (ex[i] >= 0) {
      const int r = wh[ex[i]] + rank[i];
      const int prow = s_poff[ex[i]] + r, pos = s_off[ex[i]] + r;
      slot_row[s] = prow;
      row_slot[prow] = static_cast<int>(s);
      if (order != nullptr) order[pos] = static_cast<int>(s);
      if (slot_pos != nullptr) slot_pos[s] = pos;
    } else if (s < M) {
      // an expert index outside [0, E) (the status word was raised): the slot owns no row.  -1 makes the
      // consumers of these tables skip it instead of following whatever the buffer held.
      slot_row[s] = -1;
      if (slot_pos != nullptr) slot_pos[s] = -1;
    }
  }
}

template <int W, int PL>
static int launch_permute(const long long* idx, long long M, int E, int* hist, int* counts, int* offs, int* poffs,
                          int* slot_row, int* row_slot, int* tile_expert, int* order, int* slot_pos, int* counts_out,
                          long long* load, int* status, cudaStream_t st) {
  constexpr int run = 32 * W * PL;
  const int blocks = M > run ? static_cast<int>((M + run - 1) / run) : 1;
  if (blocks > 1) {
    B200_LAUNCH((permute_hist_kernel<W, PL>), blocks, 32 * W, 0, st, idx, M, E, hist);
  }
  B200_LAUNCH((permute_rank_kernel<W, PL>), blocks, 32 * W, sizeof(int) * W * E, st, idx, M, E, hist, counts, offs, poffs,
              slot_row, row_slot, tile_expert, order, slot_pos, counts_out, load, status);
  return 0;
}

// x_s[r] = x[row_slot[r] / k] (16-byte vectors), zero rows for pads; rows >= *total_rows untouched.  Bound: the write stream
// (x stays in L2); TPR threads share a row: with a
// whole CTA a row 20 000 tokens of H 256, top-8 take 84 us (36 here), 16 384 of H 512, top-2 21 us (11 here).
template <int TPR>
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* x, const int* row_slot, const int* total_rows, int k, int vec_per_row, int pitch, uint4* x_s) {
  grid_dep_begin();
  constexpr int G = 256 / TPR;
  const int total = *total_rows;
  for (long long r = static_cast<long long>(blockIdx.x) * G + threadIdx.x / TPR; r < total;
       r += static_cast<long long>(gridDim.x) * G) {
    const int slot = row_slot[r];
    uint4* dst = x_s + r * pitch;
    const uint4* src = x + static_cast<long long>(slot / k) * vec_per_row;
    for (int c = threadIdx.x % TPR; c < vec_per_row; c += TPR) dst[c] = slot < 0 ? make_uint4(0u, 0u, 0u, 0u) : src[c];
  }
}

int permute_build(const int64_t* idx, int64_t T, int k, int E, int32_t* counts, int32_t* offs,
                  int32_t* poffs, int32_t* slot_row, int32_t* row_slot, int32_t* tile_expert,
                  int32_t* order, int32_t* slot_pos, void* ws, size_t ws_bytes,
                  int32_t* counts_out, int64_t* load, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(idx && counts && offs && poffs && slot_row && row_slot && tile_expert && ws && status,
                 B200MOE_E_NULL, "permute_build: null pointer");
  B200_CHECK_ARG(E >= 1 && E <= B200MOE_MAX_EXPERTS, B200MOE_E_UNSUPPORTED,
                 "permute_build: E = %d, supported 1..%d", E, B200MOE_MAX_EXPERTS);
  B200_CHECK_ARG(T >= 0 && k >= 1 && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE,
                 "permute_build: T = %lld, k = %d", (long long)T, k);
  const int64_t M = T * k;
  B200_CHECK_ARG(b200moe_padded_rows_cap(M, E) < (1LL << 31), B200MOE_E_BAD_SHAPE,
                 "permute_build: %lld routed rows do not fit int32 tables", (long long)M);
  B200_CHECK_ARG(ws_bytes >= b200moe_permute_ws_bytes(M, E), B200MOE_E_WS_TOO_SMALL,
                 "permute_build: workspace %zu < %zu bytes", ws_bytes, b200moe_permute_ws_bytes(M, E));
  const PermSplit split = perm_split(M);
  auto launch = split.per_lane == 16 ? launch_permute<32, 16>
                : split.warps == 8   ? launch_permute<8, 4>
                : split.warps == 16  ? launch_permute<16, 4>
                             : launch_permute<32, 4>;
  return launch(reinterpret_cast<const long long*>(idx), M, E, reinterpret_cast<int*>(ws), counts, offs, poffs, slot_row,
                row_slot, tile_expert, order, slot_pos, counts_out, reinterpret_cast<long long*>(load), status, (cudaStream_t)stream);
}

int gather_rows(const void* x, const int32_t* row_slot, const int32_t* total_rows, int k, int64_t H, int64_t ldh, int64_t rows_cap, void* x_s,
                b200moe_stream_t stream) {
  B200_CHECK_ARG(x && row_slot && total_rows && x_s, B200MOE_E_NULL, "gather_rows: null pointer");
  B200_CHECK_ARG(H > 0 && H % 8 == 0, B200MOE_E_BAD_SHAPE, "gather_rows: H = %lld must be a multiple of 8", (long long)H);
  B200_CHECK_ARG(k >= 1, B200MOE_E_BAD_SHAPE, "gather_rows: k = %d", k);
  B200_CHECK_ARG(aligned16(x) && aligned16(x_s), B200MOE_E_ALIGN, "gather_rows: pointers must be 16-byte aligned");
  if (rows_cap <= 0) return 0;
  cudaError_t err = cudaSuccess;
  by_row_threads(static_cast<int>(H / 8), [&](auto tpr) {
    constexpr int G = 256 / tpr.value;
    const long long grid = std::min<long long>((rows_cap + G - 1) / G, static_cast<long long>(num_sms()) * 16);
    err = launch_chained(gather_rows_kernel<tpr.value>, static_cast<int>(grid), 256, 0, (cudaStream_t)stream, 1,
                         reinterpret_cast<const uint4*>(x), row_slot, total_rows, k, static_cast<int>(H / 8), static_cast<int>(ldh / 8),
                         reinterpret_cast<uint4*>(x_s));
  });
  B200_CUDA(err);
  return 0;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int64_t b200moe_padded_rows_cap(int64_t M, int E) {
  if (M < 0 || E < 1) return 0;
  return ((M + B200MOE_TILE_M - 1) / B200MOE_TILE_M + E) * B200MOE_TILE_M;
}

size_t b200moe_permute_ws_bytes(int64_t M, int E) {
  if (M < 0 || E < 1) return 0;
  const int64_t nchunks = (M + 511) / 512;   // a row of E counts per 512 slots (the CTAs take at least 1024 each)
  return static_cast<size_t>((nchunks > 0 ? nchunks : 1) * E) * sizeof(int32_t);
}

int b200moe_permute_build(const int64_t* idx, int64_t T, int k, int E, int32_t* counts, int32_t* offs,
                          int32_t* poffs, int32_t* slot_row, int32_t* row_slot, int32_t* tile_expert,
                          int32_t* order, int32_t* slot_pos, void* ws, size_t ws_bytes, int32_t* status,
                          b200moe_stream_t stream) {
  return permute_build(idx, T, k, E, counts, offs, poffs, slot_row, row_slot, tile_expert, order, slot_pos, ws, ws_bytes,
                       nullptr, nullptr, status, stream);
}

int b200moe_gather_rows(const void* x, const int32_t* row_slot, const int32_t* total_rows, int k, int64_t H,
                        int64_t rows_cap, void* x_s, b200moe_stream_t stream) {
  return gather_rows(x, row_slot, total_rows, k, H, H, rows_cap, x_s, stream);
}

}  // extern "C"
