// Grouped GEMMs for few rows per expert (decoding and prompts, forward only): the WEIGHTS are the M operand of
// tcgen05.mma and the expert's rows the N operand, so the cost of a tile follows the rows an expert really has, in steps
// of 16, instead of whole 256-row tiles.
//
//   D(rows of e, N) = X(rows of e, K) * W[e](N, K)^T        computed as W[e] (128 rows of it per MMA) * X^T
//
// Bound: HBM, by the one read of the weights of the experts that have rows.  The row-tile kernels (gemm.cu) give every
// such expert a 256-row tile of MMAs, operand loads, activations and stores.  Here X lies in compact expert order
// (no pad rows), 16-row boxes of it are loaded up to the last live row, and the accumulator holds output columns in
// its lanes and rows in its columns.  A box may reach past the expert's rows: they only feed accumulator columns that
// are not stored.
// H 2048, I 1408, 64 experts, us as row tiles / here: 288 rows (4.5 an expert; 118 + 59 us at copy rate): gate/up 161 / 108, down 80 /
// 60; 9000 rows (141 an expert): 171 / 136 and 85 / 75; 6 rows of one token: 21 / 12.3 and 15 / 9.2.
// A large tile is bound by the bytes that leave L2 (weights in and out, X once per 128 columns) and wants them in flight: with a
// stage less gate/up of 9000 rows took 157 us in place of 151.  A small one is bound by latencies and by what a stage costs the
// two threads that issue it: one lane for all boxes, elected (ptx.cuh), 128-row weight boxes that hold gate and up (make_map_gate_up), and tiles of 64
// columns where even they are one wave; with a lane per box and tiles of 128 one token took 18.3 and 11.1 us.
//
// Warp roles as in gemm.cu: warp 0 TMA producer (one lane), warp 1 TMEM owner + MMA issuer, warps 2-9 epilogue.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "few_tiles.cuh"
#include "gemm_common.cuh"
#include "topk.cuh"

namespace b200moe {

struct FewParams {
  int E;
  int N;                  // output columns (SwiGLU: I)
  int K;
  const int* counts;      // rows of each expert
  const int* offs;        // first row of each expert
  void* D;                // (rows, N) bf16
  const int* act_codes;   // SwiGLU: activation code of each expert, nullptr = SiLU
  int* status;
  int aligned;            // D is 16-byte aligned
  // Counts and weights were complete when the kernel in front had passed its own wait, so before this one began (its CTAs are
  // placed after that): the first blocks of weights are loaded before the wait for that kernel, so its end and this one's start
  // cost no time on the memory bus.  That they are visible here as well is an assumption: the programming model states it past the
  // wait only.  It rests on a completed kernel's writes being in L2, where TMA reads the weights and few_tiles.cuh the counts.  Without it
  // one token takes 36.5 us instead of 35.0, 48 tokens 187.8 instead of 184.7, 1500 tokens 263 instead of 258 (64 experts of 2048 x 1408).
  int early;
};

constexpr int kFewBK = 64;      // k-block: one 128-byte swizzle row
constexpr int kFewBox = 16;     // rows of X of the small TMA box = granularity of the MMA's N
constexpr int kFewBig = 64;     // rows of the large one: a box costs the producer 45 cycles, whatever its size

// NT: most rows of one tile.  HALVES: 128-row weight blocks per stage, each with an accumulator of its own.  A SwiGLU block is 64
// gate rows and the 64 up rows of the same columns, eight and eight (make_map_gate_up).
// A CTA streams HALVES * 16 KB of weights for every live * 128 bytes of X a k-block.
template <int EPI, int NT, int HALVES>
struct FewCfg {
  static constexpr int BLOCK_COLS = EPI == EPI_SWIGLU ? 64 : 128;   // output columns of a weight block
  static constexpr int TM = BLOCK_COLS * HALVES;
  static constexpr int W_BYTES = HALVES * 128 * kFewBK * 2;
  static constexpr int X_BYTES = NT * kFewBK * 2;
  static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int ACC_COLS = HALVES * NT;                      // one tile's accumulators
  static constexpr int NBUF = 2 * ACC_COLS <= 512 ? 2 : 1;
  static constexpr int kFit = (232448 - 3072) / STAGE_BYTES;
  static constexpr int NSTAGE = kFit > 8 ? 8 : kFit;
  static constexpr int TMEM_COLS = NBUF * ACC_COLS > 256 ? 512 : NBUF * ACC_COLS > 128 ? 256 : 128;
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + (2 * NSTAGE + 2 * NBUF) * 8 + 16 + 1024;
};

template <int EPI, int NT, int HALVES>
__global__ void __launch_bounds__(kThreads, 1)
few_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                const __grid_constant__ CUtensorMap tmXbig, const FewParams p) {
  using C = FewCfg<EPI, NT, HALVES>;
  constexpr int NSTAGE = C::NSTAGE, NBUF = C::NBUF;
  constexpr int TM = C::TM;                               // output columns of a tile

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NSTAGE * C::STAGE_BYTES);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + NSTAGE);
  const uint32_t bar_tfull = smem_u32(bars + 2 * NSTAGE);
  const uint32_t bar_tempty = smem_u32(bars + 2 * NSTAGE + NBUF);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NSTAGE + 2 * NBUF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  __shared__ int pre[B200MOE_MAX_EXPERTS + 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < NBUF; ++b) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, kEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    if (NT > kFewBig) tma_prefetch_desc(&tmXbig);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  if (!p.early) grid_dep_begin();
  if (warp == 2) few_prefix<NT>(p.counts, p.E, lane, pre);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int mt = (p.N + TM - 1) / TM;
  const int total = pre[p.E] * mt;
  const int nkb = (p.K + kFewBK - 1) / kFewBK;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // One lane issues all boxes of a stage: about 210 cycles a k-block for its waits and 45 a box (measured before it was elected).
    // With a lane per box of 16 rows, the whole warp waiting, it was 510 + 54 a box: at 144 rows twice what the MMAs take.
    if (elect_one()) {
      int s = 0, ahead = 0;              // k-blocks of the first tile whose weights are on their way
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        const bool first = p.early && tile == static_cast<int>(blockIdx.x);
        const FewTile t = few_tile<NT, TM>(p.counts, p.offs, p.E, p.N, pre, tile, first);
        const int nbig = NT > kFewBig ? (t.live + kFewBox - 1) / kFewBig : 0;
        const int nsmall = max(0, (t.live - nbig * kFewBig + kFewBox - 1) / kFewBox);
        const uint32_t bytes = C::W_BYTES + nbig * (kFewBig * kFewBK * 2) + nsmall * (kFewBox * kFewBK * 2);
        auto load_w = [&](int kb, int st) {
          const uint32_t dst = smem_u32(smem + st * C::STAGE_BYTES);
          mbar_arrive_expect_tx(bar_full + 8 * st, bytes);
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            if constexpr (EPI == EPI_SWIGLU)
              tma_load_5d(dst + h * (128 * kFewBK * 2), &tmW, bar_full + 8 * st, kb * kFewBK, 0, 0, t.m0 / 8 + 8 * h, t.e);
            else
              tma_load_3d(dst + h * (128 * kFewBK * 2), &tmW, bar_full + 8 * st, kb * kFewBK, t.m0 + 128 * h, t.e);
          }
        };
        if (first) {
          ahead = min(NSTAGE, nkb);      // every stage is empty
          for (int kb = 0; kb < ahead; ++kb) load_w(kb, kb);
          grid_dep_begin();              // what X holds comes from the kernel before
        }
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, ST_WAIT_PRODUCER)) {
            ok = false;
            break;
          }
          if (kb >= ahead) load_w(kb, s);          // `ahead` is 0 after the first tile
          const uint32_t dst = smem_u32(smem + s * C::STAGE_BYTES) + C::W_BYTES;
          for (int j = 0; j < nbig; ++j)
            tma_load_3d(dst + j * (kFewBig * kFewBK * 2), &tmXbig, bar_full + 8 * s, kb * kFewBK, t.row0 + kFewBig * j, 0);
          for (int j = 0; j < nsmall; ++j)
            tma_load_3d(dst + nbig * (kFewBig * kFewBK * 2) + j * (kFewBox * kFewBK * 2), &tmX, bar_full + 8 * s, kb * kFewBK,
                        t.row0 + kFewBig * nbig + kFewBox * j, 0);
          if (++s == NSTAGE) {
            s = 0;
            ph ^= 1;
          }
        }
        ahead = 0;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (p.early) grid_dep_begin();
    if (elect_one()) {
      int s = 0, it = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, ++it) {
        const FewTile t = few_tile<NT, TM>(p.counts, p.offs, p.E, p.N, pre, tile);
        const uint32_t idesc = umma_idesc_bf16((t.live + kFewBox - 1) / kFewBox * kFewBox, 0, 0, 128);
        const int buf = it % NBUF;
        if (!mbar_wait(bar_tempty + 8 * buf, ((it / NBUF) & 1) ^ 1, abort_flag, ST_WAIT_MMA_TMEM)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * C::ACC_COLS;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, ST_WAIT_MMA_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + s * C::STAGE_BYTES);
          const uint32_t sx = sw + C::W_BYTES;
#pragma unroll
          for (int k = 0; k < kFewBK / 16; ++k) {
            const uint64_t dx = umma_desc_sw128(sx + 32 * k, 0, 1024);
#pragma unroll
            for (int h = 0; h < HALVES; ++h)
              umma_bf16(d_tmem + h * NT, umma_desc_sw128(sw + h * (128 * kFewBK * 2) + 32 * k, 0, 1024), dx, idesc,
                        (kb | k) != 0);
          }
          umma_commit(bar_empty + 8 * s);
          if (++s == NSTAGE) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        umma_commit(bar_tfull + 8 * buf);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: TMEM lane = weight row, column = row of X
    // A warp turns 16 rows of its share of a block's columns at a time, in registers, and writes 16 bytes a lane.
    const int q = warp & 3;              // TMEM lane quarter this warp may read
    const int half = (warp - 2) >> 2;    // even or odd 16-row groups
    constexpr int G = (NT + 31) / 32;    // groups of a warp, at most
    constexpr int WC = C::BLOCK_COLS / 4;                    // columns of a block in this quarter: 32, or 16 with gate and up
    if (p.early) grid_dep_begin();
    int it = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++it) {
      const FewTile t = few_tile<NT, TM>(p.counts, p.offs, p.E, p.N, pre, tile);
      const int buf = it % NBUF;
      int code = 0;
      if (EPI == EPI_SWIGLU && p.act_codes != nullptr) code = p.act_codes[t.e];
      if (!mbar_wait(bar_tfull + 8 * buf, (it / NBUF) & 1, abort_flag, ST_WAIT_EPILOGUE)) break;
      __syncwarp();
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * C::ACC_COLS;
      // bf16 values of one group, rounded before the activation as where gate and up are stored; a 16-lane block of a SwiGLU
      // tile is 8 columns of gate (v[h][2b]) and the same of up (v[h][2b + 1])
      auto fetch = [&](int hb, int c, uint32_t (&v)[2][4]) { few_fetch(taddr + hb * NT + c, v); };
      auto put = [&](auto tag, int hb, int c, const uint32_t (&v)[2][4]) {
        // 16-byte pieces: 8 output columns (piece) of a row of X
        auto write = [&](int row, int piece, uint32_t (&w)[4]) {
          const int col = t.m0 + C::BLOCK_COLS * hb + WC * q + 8 * piece;
          if (row >= t.live || col >= p.N) return;
          __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + static_cast<long long>(t.row0 + row) * p.N + col;
          if (p.aligned) {
            *reinterpret_cast<uint4*>(d) = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) reinterpret_cast<uint16_t*>(d)[i] = static_cast<uint16_t>(w[i >> 1] >> (16 * (i & 1)));
          }
        };
        const int j = lane & 3;
        if constexpr (EPI == EPI_SWIGLU) {      // two pieces, two blocks of 8 rows
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int h = i & 1, b = i >> 1;
            const float2 g = unpack_bf16x2(v[h][2 * b]), u = unpack_bf16x2(v[h][2 * b + 1]);
            constexpr int CODE = decltype(tag)::value;
            w[i] = movmatrix_trans(pack_bf16x2(glu_fwd_val<CODE>(g.x, u.x), glu_fwd_val<CODE>(g.y, u.y)));
          }
          quad_transpose(w, lane);
          write(c + 8 * (j >> 1) + (lane >> 2), j & 1, w);
        } else {                                // four pieces a block of 8 rows
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            uint32_t w[4];
            few_turn(v, b, lane, w);
            write(c + 8 * b + (lane >> 2), j, w);
          }
        }
      };
      auto by_code = [&](auto f) {       // uniform over the tile
        if (EPI == EPI_SWIGLU && code == 1) f(std::integral_constant<int, 1>());
        else if (EPI == EPI_SWIGLU && code == 5) f(std::integral_constant<int, 5>());
        else f(std::integral_constant<int, 0>());
      };
      // The only accumulators of a plain product are drained before anything else, so that the MMAs go on (9000 rows, us: 90 / 88).
      // Gate and up are not: their 96 words a thread beside the activations do not fit its registers (gate/up of 9000 rows 164 us,
      // spilled; 146 as here, and drained one block at a time 147).
      if constexpr (NBUF == 1 && EPI == EPI_STORE) {
        uint32_t v[G][HALVES][2][4];
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (16 * half + 32 * g < t.live)
#pragma unroll
            for (int hb = 0; hb < HALVES; ++hb) fetch(hb, 16 * half + 32 * g, v[g][hb]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * buf);
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (16 * half + 32 * g < t.live)
#pragma unroll
            for (int hb = 0; hb < HALVES; ++hb) put(std::integral_constant<int, 0>(), hb, 16 * half + 32 * g, v[g][hb]);
      } else {
        by_code([&](auto tag) {
#pragma unroll 1
          for (int c = 16 * half; c < t.live; c += 32)
#pragma unroll
            for (int hb = 0; hb < HALVES; ++hb) {
              uint32_t v[2][4];
              fetch(hb, c, v);
              put(tag, hb, c, v);
            }
        });
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * buf);
      }
    }
  }

  // ------------------------------------------------------------------ tear-down
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_flag);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------- router of a small batch
// Logits and top-k of 16 tokens per CTA in one launch: the gate weights are the M operand (up to 128 experts), the tokens the
// N operand; the epilogue warps hand the bf16-rounded logits over through shared memory and each picks for two tokens.
// Same k order, so the same logits to the bit, as the GEMM for large batches.  Bound by the issue of its loads and MMAs (H 2048: 128
// MMAs of 28 cycles or more, one CTA per 16 tokens) and by launch, top-k and tear-down around them: two k-blocks a stage, one elected
// thread each for loads and MMAs, a warp per token for the picks.
// us, top-6 of 64 experts at H 2048: 1 token 8.1, 48 tokens 8.4, 1500 tokens 8.9 (one k-block a stage, two lanes loading, two tokens a
// warp: 12.9, 14.4, 14.8; GEMM and top-k as two launches 15.0 ... 16.0); 64 tokens, 8 experts at H 4096 22.9 -> 12.6.  Past one wave of
// CTAs, 2368 tokens, the two launches are the faster ones (4096 tokens 17.2).
// (Dot products on CUDA cores took 5.6 us for 1 to 148 tokens, but they add in another order: about one token in ten
// thousand then takes another expert of two that are a rounding apart.)
struct RouterFewParams {
  int T, H, E, k, norm;
  float scale;
  const float* bias;
  __nv_bfloat16* logits;
  long long* idx;
  float* w;
  int* counts;
  int* status;
};

constexpr int kRouterTokens = 16;
constexpr int kRouterExperts = 128;     // at most: the lanes of one accumulator
constexpr int kRouterThreads = 64 + 32 * kRouterTokens;   // a warp per token picks

struct RouterFewCfg {
  static constexpr int KB = 2;          // k-blocks a stage
  static constexpr int W_BYTES = kRouterExperts * kFewBK * 2;
  static constexpr int KB_BYTES = W_BYTES + kRouterTokens * kFewBK * 2;
  static constexpr int STAGE_BYTES = KB * KB_BYTES;
  static constexpr int NSTAGE = 5;
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + (2 * NSTAGE + 1) * 8 + 16 + 1024;
};

template <int VPL>
__global__ void __launch_bounds__(kRouterThreads, 1)
router_few_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const RouterFewParams p) {
  using C = RouterFewCfg;
  constexpr int NSTAGE = C::NSTAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NSTAGE * C::STAGE_BYTES);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + NSTAGE);
  const uint32_t bar_done = smem_u32(bars + 2 * NSTAGE);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NSTAGE + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  __shared__ float s_logit[kRouterTokens][kRouterExperts + 1];
  __shared__ int hist[kRouterExperts];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * kRouterTokens;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) hist[e] = 0;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 32);
    tmem_relinquish();
  }
  grid_dep_begin();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int nkb = (p.H + kFewBK - 1) / kFewBK;

  if (warp == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      for (int kb = 0; kb < nkb; kb += C::KB) {
        const int n = min(C::KB, nkb - kb);
        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, ST_WAIT_PRODUCER)) break;
        mbar_arrive_expect_tx(bar_full + 8 * s, n * (p.E + kRouterTokens) * kFewBK * 2);
        for (int i = 0; i < n; ++i) {
          const uint32_t dst = smem_u32(smem + s * C::STAGE_BYTES + i * C::KB_BYTES);
          tma_load_3d(dst, &tmW, bar_full + 8 * s, (kb + i) * kFewBK, 0, 0);
          tma_load_3d(dst + C::W_BYTES, &tmX, bar_full + 8 * s, (kb + i) * kFewBK, t0, 0);
        }
        if (++s == NSTAGE) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(kRouterTokens, 0, 0, 128);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int kb = 0; kb < nkb; kb += C::KB) {
        const int n = min(C::KB, nkb - kb);
        if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, ST_WAIT_MMA_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int i = 0; i < n; ++i) {
          const uint32_t sw = smem_u32(smem + s * C::STAGE_BYTES + i * C::KB_BYTES);
#pragma unroll
          for (int k = 0; k < kFewBK / 16; ++k)
            umma_bf16(tmem_base, umma_desc_sw128(sw + 32 * k, 0, 1024), umma_desc_sw128(sw + C::W_BYTES + 32 * k, 0, 1024),
                      idesc, (kb | i | k) != 0);
        }
        umma_commit(bar_empty + 8 * s);
        if (++s == NSTAGE) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok) umma_commit(bar_done);
    }
  } else {
    const int ew = warp - 2, q = warp & 3;     // TMEM lane quarter; the first four warps read the accumulator
    float b[VPL];                              // on its way while the products run
#pragma unroll
    for (int i = 0; i < VPL; ++i) b[i] = (p.bias != nullptr && lane + 32 * i < p.E) ? p.bias[lane + 32 * i] : 0.0f;
    const bool ok = mbar_wait(bar_done, 0, abort_flag, ST_WAIT_EPILOGUE);
    __syncwarp();
    tc_fence_after();
    if (ok && ew < 4) {
      uint32_t a[kRouterTokens];
      tmem_ld16(tmem_base + (static_cast<uint32_t>(q * 32) << 16), a);
      tmem_ld_wait();
#pragma unroll
      for (int t = 0; t < kRouterTokens; ++t) s_logit[t][32 * q + lane] = bf16_round(__uint_as_float(a[t]));
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kRouterTokens) : "memory");    // the epilogue warps only
    const long long t = t0 + ew;
    if (ok && t < p.T) {
      float sc[VPL];
      uint32_t key[VPL];
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int e = lane + 32 * i;
        sc[i] = 0.0f;
        key[i] = 0u;
        if (e < p.E) {
          const float v = s_logit[ew][e];
          p.logits[t * p.E + e] = __float2bfloat16_rn(v);
          sc[i] = sigmoid_f(v);
          key[i] = select_key(sc[i] + b[i]);
        }
      }
      int my_idx;
      float my_w;
      topk_of_token<VPL>(sc, key, p.k, p.norm, p.scale, hist, p.counts != nullptr, my_idx, my_w);
      if (lane < p.k) {
        p.idx[t * p.k + lane] = my_idx;
        p.w[t * p.k + lane] = my_w;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (p.counts != nullptr)
    for (int e = threadIdx.x; e < p.E; e += blockDim.x)
      if (hist[e] != 0) atomicAdd(&p.counts[e], hist[e]);
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_flag);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 32);
  }
}

// ---------------------------------------------------------------------------- host side
template <int EPI, int NT, int HALVES>
static int launch_few(const void* x, const void* w, int64_t rows_cap, const FewParams& p, cudaStream_t stream) {
  using C = FewCfg<EPI, NT, HALVES>;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(few_rows_kernel<EPI, NT, HALVES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    C::SMEM_BYTES);
  });
  if (attr_err != cudaSuccess) return cuda_fail(attr_err, "cudaFuncSetAttribute(max dynamic smem)");
  CUtensorMap tmW, tmX, tmXbig;
  int rc = EPI == EPI_SWIGLU ? make_map_gate_up(&tmW, w, p.K, p.N, p.E, 8)
                             : make_map(&tmW, w, p.K, p.N, p.E, p.K, static_cast<uint64_t>(p.N) * p.K, kFewBK, 128);
  if (rc) return rc;
  rc = make_map(&tmX, x, p.K, rows_cap, 1, p.K, static_cast<uint64_t>(rows_cap) * p.K, kFewBK, kFewBox);
  if (rc) return rc;
  tmXbig = tmX;
  if (NT > kFewBig) rc = make_map(&tmXbig, x, p.K, rows_cap, 1, p.K, static_cast<uint64_t>(rows_cap) * p.K, kFewBK, kFewBig);
  if (rc) return rc;
  const long long chunks = std::min<long long>(rows_cap, p.E + rows_cap / NT);   // at most
  const long long tiles = chunks * ceil_div(p.N, C::TM);
  const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>(gemm_cta_budget(), tiles)));
  B200_LAUNCH((few_rows_kernel<EPI, NT, HALVES>), grid, kThreads, C::SMEM_BYTES, stream, tmW, tmX, tmXbig, p);
  return 0;
}

template <int VPL>
static int launch_router_few(const void* x, const void* weight, const RouterFewParams& p, cudaStream_t stream) {
  using C = RouterFewCfg;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(router_few_kernel<VPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  });
  if (attr_err != cudaSuccess) return cuda_fail(attr_err, "cudaFuncSetAttribute(max dynamic smem)");
  CUtensorMap tmW, tmX;   // a weight box of E rows: what the MMA reads past them ends in lanes nobody reads
  int rc = make_map(&tmW, weight, p.H, p.E, 1, p.H, static_cast<uint64_t>(p.E) * p.H, kFewBK, p.E);
  if (rc) return rc;
  rc = make_map(&tmX, x, p.H, p.T, 1, p.H, static_cast<uint64_t>(p.T) * p.H, kFewBK, kRouterTokens);
  if (rc) return rc;
  B200_LAUNCH(router_few_kernel<VPL>, (p.T + kRouterTokens - 1) / kRouterTokens, kRouterThreads, C::SMEM_BYTES, stream, tmW, tmX, p);
  return 0;
}

// Tile.  The host knows the mean rows per expert, not the counts: both rules below were timed under even routing, expert
// frequencies ~ rank^-0.6 and rank^-1.1, and one expert in every token's picks.  us of gate/up + down with permutation, gather
// and combine, L2 flushed before each.
//  - Chunks of 64 rows where even the worst spread of the rows over the experts, E + M / 64 chunks, is one wave of CTAs: the
//    smallest tile then has the shortest chain and the most SMs.  8 experts, 512 x 256, mean 140 rows, even / rank^-1.1:
//    NT 64 30 / 30, 128 34 / 34, 192 38 / 40 (row tiles 34 / 34).
//  - Else by the mean.  A larger NT keeps an expert's rows in one tile, so its weights pass through shared memory once; a
//    smaller one leaves room for more k-blocks in flight and double-buffered accumulators.  64 experts, 2048 x 1408, even /
//    rank^-1.1: mean 4 rows NT 64 197 / 164, 128 200 / 166, 192 201 / 164; 39 rows 211 / 217, 211 / 217, 211 / 211; 80 rows
//    252 / 246, 221 / 232, 221 / 227; 110 rows 266 / 291, 229 / 257, 231 / 246; 140 rows 345 / 340, 285 / 274, 245 / 268.
//    kFewRows128 stands where an NT 192 that spilled put it: between 40 and 110 rows the two are now within 2 % under even
//    routing and NT 192 leads under a skewed one, most with few experts (8 of 4096 x 14336, 80 rows 594 against 520).
constexpr int64_t kFewRows64 = 40, kFewRows128 = 110;

static int64_t few_blocks(int64_t N, int64_t K) { return ceil_div(std::max(N, K), 128); }   // weight blocks of an expert (either product)
static bool few_one_wave(int64_t M, int E, int64_t N, int64_t K) { return (E + M / 64) * few_blocks(N, K) <= num_sms(); }

static int few_nt(int64_t M, int E, int64_t N, int64_t K) {
  if (M <= kFewRows64 * E || few_one_wave(M, E, N, K)) return 64;
  return M <= kFewRows128 * E ? 128 : 192;
}

// Gate/up blocks of 64 columns instead of 128, where even they are one wave: half the chain of a tile, twice the SMs that stream.
static bool few_narrow(int64_t M, int E, int64_t I) {
  return (std::min<int64_t>(E, M) + M / 64) * ceil_div(I, 64) <= num_sms();
}

// Whether a forward without a backward runs over compact rows (this file) or row tiles (gemm.cu), same measurements, row tiles
// against compact rows, even / rank^-1.1.  64 experts, 2048 x 1408: mean 4 rows 274 / 225 against 197 / 164, 140 rows 289 /
// 330 against 245 / 268, 200 rows 304 / 386 against 342 / 325 (an even expert then takes two tiles): up to kFewRows.
// Fewer than 16 experts leave few pad rows in row tiles: 8 experts, 4096 x 14336: 80 rows 586 / 608 against 492 / 596, 110 rows
// 610 / 746 against 520 / 709: up to kFewRows128.  Both limits on few experts were drawn with a slower NT 192 and now give some
// away: 159 rows there 618 / 841 against 534 / 726, and where one chunk per expert fills less than half of the SMs and the
// chunks of 64 are more than one wave, 8 experts of 1024 x 1024, 140 rows 56 / 49 against 46 / 41 (NT 128).
// Every token's one pick on one expert, the spread the host cannot see: 16 experts, 4096 x 1024, 39 rows on average 76 against
// 72, 60 rows 61 against 59, 159 rows 102 against 90.
constexpr int64_t kFewRows = 160;

bool few_rows_forward(int64_t M, int E, int64_t H, int64_t I) {
  if (M > kFewRows * E) return false;
  if (few_one_wave(M, E, H, I)) return true;
  if (E * few_blocks(H, I) <= num_sms() / 2) return false;
  return E >= 16 || M <= kFewRows128 * E;
}

static int check_few(const char* who, const void* x, const void* w, const void* d, const int32_t* counts,
                     const int32_t* offs, int64_t rows_cap, int E, int64_t N, int64_t K) {
  B200_CHECK_ARG(x && w && d && counts && offs, B200MOE_E_NULL, "%s: null pointer", who);
  B200_CHECK_ARG(E >= 1 && E <= B200MOE_MAX_EXPERTS, B200MOE_E_UNSUPPORTED, "%s: E = %d, supported 1..%d", who, E,
                 B200MOE_MAX_EXPERTS);
  B200_CHECK_ARG(rows_cap > 0 && rows_cap < (1LL << 31), B200MOE_E_BAD_SHAPE, "%s: rows_cap = %lld", who, (long long)rows_cap);
  B200_CHECK_ARG(N > 0 && N % 8 == 0 && K > 0 && K % 8 == 0, B200MOE_E_BAD_SHAPE,
                 "%s: N = %lld and K = %lld must be positive multiples of 8", who, (long long)N, (long long)K);
  B200_CHECK_ARG(N < (1LL << 31) && K < (1LL << 31), B200MOE_E_BAD_SHAPE, "%s: extent beyond 2^31", who);
  return 0;
}

int expert_gate_up_few(const void* x, const void* gate_up_proj, const int32_t* act_codes, const int32_t* counts,
                       const int32_t* offs, int64_t rows_cap, int E, int64_t H, int64_t I, int early, void* inter,
                       int32_t* status, b200moe_stream_t stream) {
  int rc = check_few("expert_gate_up_few", x, gate_up_proj, inter, counts, offs, rows_cap, E, I, H);
  if (rc) return rc;
  FewParams p{E, static_cast<int>(I), static_cast<int>(H), counts, offs, inter, act_codes, status, aligned16(inter), early};
  cudaStream_t st = (cudaStream_t)stream;
  const int nt = few_nt(rows_cap, E, I, H);
  if (nt == 64 && few_narrow(rows_cap, E, I)) return launch_few<EPI_SWIGLU, 64, 1>(x, gate_up_proj, rows_cap, p, st);
  if (nt == 64) return launch_few<EPI_SWIGLU, 64, 2>(x, gate_up_proj, rows_cap, p, st);
  if (nt == 128) return launch_few<EPI_SWIGLU, 128, 2>(x, gate_up_proj, rows_cap, p, st);
  return launch_few<EPI_SWIGLU, 192, 2>(x, gate_up_proj, rows_cap, p, st);
}

int expert_linear_few(const void* x, const void* w, const int32_t* counts, const int32_t* offs, int64_t rows_cap, int E,
                      int64_t N, int64_t K, int early, void* out, int32_t* status, b200moe_stream_t stream) {
  int rc = check_few("expert_linear_few", x, w, out, counts, offs, rows_cap, E, N, K);
  if (rc) return rc;
  FewParams p{E, static_cast<int>(N), static_cast<int>(K), counts, offs, out, nullptr, status, aligned16(out), early};
  cudaStream_t st = (cudaStream_t)stream;
  const int nt = few_nt(rows_cap, E, N, K);
  if (nt == 64) return launch_few<EPI_STORE, 64, 1>(x, w, rows_cap, p, st);
  if (nt == 128) return launch_few<EPI_STORE, 128, 1>(x, w, rows_cap, p, st);
  return launch_few<EPI_STORE, 192, 2>(x, w, rows_cap, p, st);
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_expert_gate_up_few(const void* x, const void* gate_up_proj, const int32_t* act_codes, const int32_t* counts,
                               const int32_t* offs, int64_t rows_cap, int E, int64_t H, int64_t I, void* inter,
                               int32_t* status, b200moe_stream_t stream) {
  return expert_gate_up_few(x, gate_up_proj, act_codes, counts, offs, rows_cap, E, H, I, 0, inter, status, stream);
}

int b200moe_expert_linear_few(const void* x, const void* w, const int32_t* counts, const int32_t* offs, int64_t rows_cap,
                              int E, int64_t N, int64_t K, void* out, int32_t* status, b200moe_stream_t stream) {
  return expert_linear_few(x, w, counts, offs, rows_cap, E, N, K, 0, out, status, stream);
}

int b200moe_router_small_fwd(const void* x, const void* weight, const float* bias, int64_t T, int64_t H, int E, int k,
                             int norm_topk, float scale, void* logits, int64_t* idx, float* w, int32_t* counts,
                             int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(x && weight && logits && idx && w, B200MOE_E_NULL, "router_small_fwd: null pointer");
  B200_CHECK_ARG(E >= 1 && E <= kRouterExperts, B200MOE_E_UNSUPPORTED, "router_small_fwd: E = %d, supported 1..%d", E,
                 kRouterExperts);
  B200_CHECK_ARG(E % 8 == 0 && H > 0 && H % 8 == 0, B200MOE_E_BAD_SHAPE,
                 "router_small_fwd: E = %d and H = %lld must be positive multiples of 8", E, (long long)H);
  B200_CHECK_ARG(k >= 1 && k <= E && k <= B200MOE_MAX_TOPK, B200MOE_E_BAD_SHAPE,
                 "router_small_fwd: top_k = %d must be in 1..min(E=%d, %d)", k, E, B200MOE_MAX_TOPK);
  B200_CHECK_ARG(T >= 0 && T < (1LL << 31) && H < (1LL << 31), B200MOE_E_BAD_SHAPE, "router_small_fwd: T = %lld", (long long)T);
  cudaStream_t st = (cudaStream_t)stream;
  if (counts != nullptr) B200_CUDA(cudaMemsetAsync(counts, 0, sizeof(int32_t) * E, st));
  if (T == 0) return 0;
  RouterFewParams p{static_cast<int>(T), static_cast<int>(H), E, k, norm_topk, scale, bias, reinterpret_cast<__nv_bfloat16*>(logits),
                    reinterpret_cast<long long*>(idx), w, counts, status};
  if (E <= 32) return launch_router_few<1>(x, weight, p, st);
  if (E <= 64) return launch_router_few<2>(x, weight, p, st);
  return launch_router_few<4>(x, weight, p, st);
}

}  // extern "C"
