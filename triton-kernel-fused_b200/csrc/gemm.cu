// Persistent bf16 GEMM for sm_100a: TMA -> 128B-swizzled shared-memory ring -> tcgen05.mma with the
// fp32 accumulator in TMEM (double buffered) -> epilogue warps read TMEM and store.
//
// One kernel serves every contraction of the MoE block:
//   schedule  DENSE      D(M,N)            = A * B          (router projections)
//             GROUPED_M  D(rows of e, N)   = A(rows of e) * B[e]   (expert forward + dgrad)
//             GROUPED_K  D[e](M,N)         = A(rows of e)^T * B(rows of e)   (expert wgrad, split-K)
//   operand majors: K-major (reduction index contiguous) or MN-major (row/column index contiguous)
//   epilogues: bf16 store, SwiGLU (gate|up -> gate_up + inter), GLU backward, fp32 store.
//   CTAS = 1: one CTA computes a 128 x BN tile.
//   CTAS = 2: a CTA pair (cluster of 2) computes a 256 x 256 tile with tcgen05 cta_group::2: each CTA
//             stages its own 128 rows of A and its own 128 columns of B, the leader CTA issues the
//             MMAs for both, each CTA's TMEM holds its 128 rows of the accumulator.  This halves
//             the L2 -> shared-memory traffic per FLOP and leaves room for 6 stages instead of 4.
//
// Warp roles (320 threads, 352 with single-CTA tiles): warp 0 = TMA producer and warp 1 = TMEM owner + MMA issuer (an elected
// thread each), warp 10 = TMA producer of B (single-CTA tiles only), warps 2-9 = epilogue (TMEM lane quarter = warp_id % 4, two warps per quarter split the
// columns).
#include <cuda.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gemm_common.cuh"

namespace b200moe {

constexpr int BK = 64;   // k-block: 64 bf16 = one 128-byte swizzle row

// BN = 256 kernels with a bf16 result stage it in shared memory and write it with TMA stores
template <int BN, int EPI>
__host__ __device__ constexpr bool tma_epilogue() { return BN == 256 && EPI != EPI_STORE_F32; }

// EPI_WARP_BYTES: shared memory each epilogue warp owns (0: none, 4 KB: one output staging box,
// 8 KB: the GLU-backward gate and up boxes that are loaded by TMA and overwritten in place)
constexpr int kGluBoxBytes = 32 * 64;   // GLU backward: one 32 rows x 32 columns bf16 box

template <int BN, int EPI>
__host__ __device__ constexpr int epi_warp_bytes() {
  return !tma_epilogue<BN, EPI>() ? 0 : (EPI == EPI_GLU_BWD ? 2 * kStageOutBytes : kStageOutBytes);
}

template <int BN, int CTAS, int EPI_WARP_BYTES = 0>
struct Cfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = (BN / CTAS) * BK * 2;   // per CTA
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_BYTES = kEpiWarps * EPI_WARP_BYTES;
  static constexpr int kBudget = 232448 - 1024 - 256;       // 227 KB minus alignment slack and barriers
  static constexpr int kFit = (kBudget - EPI_BYTES) / STAGE_BYTES;
  static constexpr int NSTAGE = kFit > 8 ? 8 : kFit;
  static constexpr int TMEM_COLS = 2 * BN;  // two accumulators; 128, 256 or 512 (power of two >= 32)
  static constexpr int BAR_BYTES = (2 * NSTAGE + 4 + 2 * kEpiWarps) * 8 + 16;
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + EPI_BYTES + BAR_BYTES + 1024;  // + alignment slack
  static constexpr int TILE_ROWS = BM * CTAS;
};

// Columns of B (and of the accumulator) a pair tile multiplies: the last tile of a ragged width is narrower, in steps of 32
// with K-major weights (the two-SM MMA with 256 rows takes an N that is a multiple of 32; a CTA's half of B then is whole
// 8-row groups of its shared-memory layout), of 128 with MN-major ones (a 64-wide swizzle atom per CTA).  SwiGLU tiles stay
// whole: a narrow one gained nothing on ragged widths, and the epilogue's variable offset of the up columns cost 1 % on the
// others.  This is what lets every width above 64 take the pair kernel: its 256-wide tiles
// multiply no more columns than 128-wide single-CTA tiles would, at half the operand traffic per FLOP.  One layer of
// 3001 tokens, H 1032, I 680, 32 experts, top-4: the five products that ran on 128-wide tiles 321 -> 228 us.
__host__ __device__ constexpr int pair_width(int rem, bool b_mn, int bn) {
  return b_mn ? (rem <= bn / 2 ? bn / 2 : bn) : (rem >= bn ? bn : (rem + 31) / 32 * 32);
}
constexpr bool pair_widths_valid(int bn) {
  for (int rem = 1; rem <= 2 * bn; ++rem)
    for (int mn = 0; mn < 2; ++mn) {
      const int w = pair_width(rem, mn != 0, bn);
      if (w % 32 != 0 || w < 32 || w > bn || w < (rem < bn ? rem : bn)) return false;
    }
  return true;
}
static_assert(pair_widths_valid(256), "a pair tile's N must cover its columns and be a multiple of 32 up to 256");

template <int BN, int EPI>
__device__ __forceinline__ int pair_cols(const GemmParams& p, int n0) {
  if constexpr (EPI == EPI_SWIGLU) return BN;
  return pair_width(p.N - n0, p.b_mn != 0, BN);
}

// POLY: the variant of the kernel.  GLU epilogues: per-expert activation codes 0 / 1 / 5 (p.act_codes); false =
// SiLU for every expert.  Store epilogues (EPI_STORE, EPI_STORE_F32): a convolution operand (p.conv_taps), compiled
// only into the instantiations the conv-router entry points launch, so that the expert GEMMs carry no code for it.
// Single-CTA tiles have two loading warps, one for A and one for B: a k-block's MMAs take 256 cycles there, but one thread's wait, its two
// boxes and a convolution's coordinates 480 (380 without those), whatever the batch.  Logits of 16 x 1024 positions of H 2048, 64 experts, 4
// taps (us): one loading warp 35.7, two 29.8, the next stage's barrier asked for ahead 28.6, the convolution in a loop of its own 24.7; of
// 1 x 1024 positions 34.2 -> 23.4.  Products of few k-blocks are as fast as before.
__host__ __device__ constexpr int gemm_threads(int ctas) { return ctas == 1 ? kThreads + 32 : kThreads; }

template <int BN, int EPI, int CTAS, bool POLY = false>
__global__ void __launch_bounds__(gemm_threads(CTAS), 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmD2,
            const GemmParams p) {
  constexpr bool TMA_EPI = tma_epilogue<BN, EPI>();
  using C = Cfg<BN, CTAS, epi_warp_bytes<BN, EPI>()>;
  constexpr int TN = (EPI == EPI_SWIGLU) ? BN / 2 : BN;   // output columns one tile covers
  constexpr int TM = C::TILE_ROWS;
  constexpr int NSTAGE = C::NSTAGE;
  constexpr int BNC = BN / CTAS;                          // B columns staged by one CTA
  constexpr bool kPeek = CTAS == 1;                       // the next stage's barrier is asked for while this one's boxes / MMAs go out

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* epi_smem = smem + NSTAGE * C::STAGE_BYTES;   // 1024-aligned: stages are multiples of 8 KB
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + C::EPI_BYTES);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + NSTAGE);
  const uint32_t bar_tfull = smem_u32(bars + 2 * NSTAGE);
  const uint32_t bar_tempty = smem_u32(bars + 2 * NSTAGE + 2);
  const uint32_t bar_epi = smem_u32(bars + 2 * NSTAGE + 4);   // two per epilogue warp (GLU backward load sets)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NSTAGE + 4 + 2 * kEpiWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = (CTAS == 2) ? cluster_ctarank() : 0u;   // 0 = leader of the pair
  const int first_tile = (CTAS == 2) ? static_cast<int>(cluster_id_x()) : static_cast<int>(blockIdx.x);
  const int tile_step = (CTAS == 2) ? static_cast<int>(num_clusters_x()) : static_cast<int>(gridDim.x);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, kEpiWarps * CTAS);
    }
    for (int w = 0; w < 2 * kEpiWarps; ++w) mbar_init(bar_epi + 8 * w, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    if constexpr (CTAS == 2) {
      tmem_alloc_pair(smem_u32(tmem_slot), C::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
      tmem_relinquish();
    }
  }
  __shared__ int s_order[B200MOE_MAX_EXPERTS];
  grid_dep_wait();
  const int* order = build_group_order(p, s_order);
  tc_fence_before();
  __syncthreads();
  if constexpr (CTAS == 2) {   // peer barriers are initialised before any remote arrive
    __syncwarp();
    cluster_sync_all();
  }
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  constexpr bool WINDOW = (EPI == EPI_SWIGLU || EPI == EPI_GLU_BWD);   // entry points with a row window
  constexpr bool CONV = POLY && (EPI == EPI_STORE || EPI == EPI_STORE_F32);   // launched by the conv-router entry points
  const int total = total_tiles(p, TN, TM, WINDOW);
  const int row_base = (WINDOW && p.row_hi > 0) ? p.row_lo : 0;

  if (warp == 0 || warp >= 2 + kEpiWarps) {
    // ------------------------------------------------------------------ TMA producer (each CTA)
    auto produce = [&](auto do_a, auto do_b) {
      constexpr bool A = do_a.value, B = do_b.value;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true, ready = false;
      for (int tile = first_tile; tile < total && ok; tile += tile_step) {
        const Tile t = get_tile(p, tile, TN, TM, 64, order, row_base, CONV);
        const int gB = (p.sched == SCHED_GROUPED_M) ? t.g : 0;
        const int m0 = t.m0 + BM * static_cast<int>(cta_rank);
        // a narrower last pair tile: each CTA supplies half of its columns of B, the first ones of its (still
        // BN/2 wide) staging tile
        [[maybe_unused]] const int bstep = (CTAS == 2) ? pair_cols<BN, EPI>(p, t.n0) / 2 : BNC;
        // coordinates of the B boxes; a convolution operand (see GemmParams::conv_taps) replaces the flat row by (position + shift,
        // batch).  Its divisions are done once per tile, the k-loop only counts.
        int b_n0 = t.n0, b_k = t.k0, b_g = gB;
        if (CONV && p.conv_taps > 0 && p.sched != SCHED_DENSE) {
          const int tap = t.n0 / p.conv_C;
          b_n0 = t.n0 - tap * p.conv_C;
          b_g = t.k0 / p.conv_S;
          b_k = t.k0 - b_g * p.conv_S + tap - (p.conv_taps - 1);
        }
        if constexpr (CONV && CTAS == 1)
          if (p.conv_taps > 0 && p.sched == SCHED_DENSE) {       // tap by tap, with nothing in the loop but its box
            const int pos0 = m0 - p.conv_sign * (p.conv_taps - 1);
            for (int tap = 0; tap < p.conv_taps && ok; ++tap) {
              for (int c0 = 0; c0 < p.conv_C; c0 += BK) {
                if (!ready && !mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, ST_WAIT_PRODUCER)) {
                  ok = false;
                  break;
                }
                const uint32_t full = bar_full + 8 * s, sa = smem_u32(smem + s * C::STAGE_BYTES);
                if (++s == NSTAGE) {
                  s = 0;
                  ph ^= 1;
                }
                ready = mbar_test_wait(bar_empty + 8 * s, ph ^ 1);
                if constexpr (A) {
                  mbar_arrive_expect_tx(full, C::STAGE_BYTES);
                  tma_load_3d(sa, &tmA, full, c0, pos0 + p.conv_sign * tap, t.g);
                }
                if constexpr (B) {
                  const uint32_t sb = sa + C::A_BYTES;
                  if (!p.b_mn) {
                    tma_load_3d(sb, &tmB, full, p.conv_b_taps ? c0 : tap * p.conv_C + c0, t.n0, p.conv_b_taps ? tap : 0);
                  } else {
#pragma unroll
                    for (int j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * (64 * BK * 2), &tmB, full, t.n0 + 64 * j, tap * p.conv_C + c0, 0);
                  }
                }
              }
            }
            continue;
          }
        for (int kb = 0; kb < t.nkb; ++kb) {
          if (!ready && !mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, ST_WAIT_PRODUCER)) {
            ok = false;
            break;
          }
          if constexpr (kPeek) ready = mbar_test_wait(bar_empty + (s + 1 == NSTAGE ? 0 : 8 * (s + 1)), s + 1 == NSTAGE ? ph : ph ^ 1);
          const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES);
          const uint32_t sb = sa + C::A_BYTES;
          const int kk = t.k0 + kb * BK;
          if (!CONV || p.conv_taps == 0) b_k = kk;
          if constexpr (CTAS == 1) {
            const uint32_t full = bar_full + 8 * s;
            if constexpr (A) mbar_arrive_expect_tx(full, C::STAGE_BYTES);
            if (!A) {
            } else if (!p.a_mn) {
              tma_load_3d(sa, &tmA, full, kk, m0, 0);  // box {64 k, 128 rows}
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j)  // boxes {64 mn, 64 k-rows}
                tma_load_3d(sa + j * (64 * BK * 2), &tmA, full, m0 + 64 * j, kk, 0);
            }
            if constexpr (!B) {
            } else if constexpr (EPI == EPI_SWIGLU) {
              // gate rows [n0, n0+BN/2) of W[e] then up rows of the same range: dims {H, I, 2E}
              tma_load_3d(sb, &tmB, full, kk, t.n0, 2 * gB);
              tma_load_3d(sb + (BN / 2) * BK * 2, &tmB, full, kk, t.n0, 2 * gB + 1);
            } else if (!p.b_mn) {
              tma_load_3d(sb, &tmB, full, kk, t.n0, b_g);  // box {64 k, BN rows}
            } else {
#pragma unroll
              for (int j = 0; j < BN / 64; ++j)
                tma_load_3d(sb + j * (64 * BK * 2), &tmB, full, b_n0 + 64 * j, b_k, b_g);
            }
          } else {
            // the leader's barrier counts the bytes of both CTAs
            const uint32_t full = mapa_shared(bar_full + 8 * s, 0);
            if (cta_rank == 0) mbar_arrive_expect_tx(bar_full + 8 * s, 2 * C::STAGE_BYTES);
            if (!p.a_mn) {
              tma_load_3d_pair(sa, &tmA, full, kk, m0, 0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j)
                tma_load_3d_pair(sa + j * (64 * BK * 2), &tmA, full, m0 + 64 * j, kk, 0);
            }
            if constexpr (EPI == EPI_SWIGLU) {
              // leader stages the gate rows, the peer the up rows of I-columns [n0, n0+128)
              tma_load_3d_pair(sb, &tmB, full, kk, t.n0, 2 * gB + static_cast<int>(cta_rank));
            } else if (!p.b_mn) {
              tma_load_3d_pair(sb, &tmB, full, kk, t.n0 + bstep * static_cast<int>(cta_rank), b_g);
            } else {
#pragma unroll
              for (int j = 0; j < BNC / 64; ++j)
                tma_load_3d_pair(sb + j * (64 * BK * 2), &tmB, full,
                                 b_n0 + bstep * static_cast<int>(cta_rank) + 64 * j, b_k, b_g);
            }
          }
          if (CONV && p.conv_taps > 0) {       // the next k-block's rows of B
            b_k += BK;
            if (kk + BK - b_g * p.conv_S >= p.conv_S) {   // next batch
              ++b_g;
              b_k -= p.conv_S;
            }
          }
          if (++s == NSTAGE) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    };
    if (elect_one()) {
      if constexpr (CTAS == 2) produce(std::true_type(), std::true_type());
      else if (warp == 0) produce(std::true_type(), std::false_type());
      else produce(std::false_type(), std::true_type());
    }
    grid_dep_launch();   // the last loads are on their way
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (cta_rank == 0 && elect_one()) {
      // K-major: rows are 128 B apart, 8-row groups 1024 B apart, 16 k-elements = 32 B.
      // MN-major: 64-wide MN blocks are 64*128 B apart (LBO), 8 k-rows 1024 B apart (SBO),
      //           16 k-rows = 2048 B.
      const uint32_t a_lbo = p.a_mn ? 64 * BK * 2 : 0, b_lbo = p.b_mn ? 64 * BK * 2 : 0;
      const uint32_t a_kstep = p.a_mn ? 2048 : 32, b_kstep = p.b_mn ? 2048 : 32;
      int s = 0, it = 0;
      uint32_t ph = 0;
      bool ok = true, ready = false;
      for (int tile = first_tile; tile < total && ok; tile += tile_step, ++it) {
        const Tile t = get_tile(p, tile, TN, TM, 64, order, row_base, CONV);
        const int buf = it & 1;
        if (!mbar_wait(bar_tempty + 8 * buf, ((it >> 1) & 1) ^ 1, abort_flag, ST_WAIT_MMA_TMEM)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        const uint32_t idesc = umma_idesc_bf16(CTAS == 2 ? pair_cols<BN, EPI>(p, t.n0) : BN, p.a_mn, p.b_mn, TM);
        for (int kb = 0; kb < t.nkb; ++kb) {
          if (!ready && !mbar_wait(bar_full + 8 * s, ph, abort_flag, ST_WAIT_MMA_FULL)) {
            ok = false;
            break;
          }
          if constexpr (kPeek) ready = mbar_test_wait(bar_full + (s + 1 == NSTAGE ? 0 : 8 * (s + 1)), s + 1 == NSTAGE ? ph ^ 1 : ph);
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES);
          const uint32_t sb = sa + C::A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = umma_desc_sw128(sa + k * a_kstep, a_lbo, 1024);
            const uint64_t db = umma_desc_sw128(sb + k * b_kstep, b_lbo, 1024);
            if constexpr (CTAS == 2) umma_bf16_pair(d_tmem, da, db, idesc, (kb | k) != 0);
            else umma_bf16(d_tmem, da, db, idesc, (kb | k) != 0);
          }
          // frees the stage (in both CTAs) when these MMAs have read it
          if constexpr (CTAS == 2) umma_commit_pair(bar_empty + 8 * s);
          else umma_commit(bar_empty + 8 * s);
          if (++s == NSTAGE) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        if (t.nkb > 0) {
          if constexpr (CTAS == 2) umma_commit_pair(bar_tfull + 8 * buf);
          else umma_commit(bar_tfull + 8 * buf);
        } else {
          mbar_arrive(bar_tfull + 8 * buf);
          if constexpr (CTAS == 2) mbar_arrive_cluster(mapa_shared(bar_tfull + 8 * buf, 1));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (8 warps per CTA)
    const int q = warp & 3;              // TMEM lane quarter this warp may read
    const int half = (warp - 2) >> 2;    // which half of the tile's columns this warp handles
    const uint32_t tempty_leader = (CTAS == 2) ? mapa_shared(bar_tempty, 0) : bar_tempty;
    uint32_t epi_phase = 0;   // parity of this warp's GLU-backward load barrier
    int it = 0;
    for (int tile = first_tile; tile < total; tile += tile_step, ++it) {
      const Tile t = get_tile(p, tile, TN, TM, 64, order, row_base, CONV);
      const int buf = it & 1;
      int act_code = 0;   // activation of this tile's expert (uniform over the tile)
      if constexpr (POLY && (EPI == EPI_SWIGLU || EPI == EPI_GLU_BWD)) act_code = p.act_codes[t.g];
      const int row0 = t.m0 + BM * static_cast<int>(cta_rank) + q * 32;   // first row of this warp
      const long long row = static_cast<long long>(row0) + lane;
      // GLU backward works on four 32-column sub-chunks per warp with two sets of (gate, up) boxes of
      // 32 rows x 32 columns (2 KB, 64-byte swizzle): a set is loaded by TMA, overwritten in place with
      // grad_gate / grad_up and stored by TMA while the other set is loading or being computed on.  The saved
      // gate/up values do not depend on the accumulator, so the first two loads go out before the MMAs of
      // the tile are waited for.
      const int glu_col0 = t.n0 + half * (BN / 2);
      uint8_t* ebuf = epi_smem + (warp - 2) * C::EPI_BYTES / kEpiWarps;   // [set][gate | up] boxes of 2 KB
      const uint32_t ebar = bar_epi + 16 * (warp - 2);                     // + 8 * set
      auto glu_load = [&](int sub) {   // tmD2 = saved gate_up seen as {I, rows, 2}, box {32, 32}
        const int set = sub & 1;
        if (lane == 0) {
          mbar_arrive_expect_tx(ebar + 8 * set, 2 * kGluBoxBytes);
          tma_load_3d(smem_u32(ebuf + set * 2 * kGluBoxBytes), &tmD2, ebar + 8 * set, glu_col0 + 32 * sub, row0, 0);
          tma_load_3d(smem_u32(ebuf + set * 2 * kGluBoxBytes + kGluBoxBytes), &tmD2, ebar + 8 * set,
                      glu_col0 + 32 * sub, row0, 1);
        }
      };
      uint8_t* bufG = ebuf;   // staging box of the other TMA-store epilogues
      if constexpr (TMA_EPI && EPI == EPI_GLU_BWD) {
        staging_free(lane);   // the previous tile's stores out of these boxes have been read
        if (glu_col0 < p.I) glu_load(0);
        if (glu_col0 + 32 < p.I) glu_load(1);
      }
      // single-CTA GLU backward: gate and up of a step (16 rows x CW columns) as they lie in memory, the first one's on their way
      // while the MMAs run, the next one's while one is computed
      constexpr int CW = (EPI == EPI_SWIGLU ? BN / 4 : BN / 2) >= 64 ? 64 : 32;      // columns at a time (epilogues without TMA)
      constexpr int NP = CW / 32;
      constexpr bool kGluRegs = !TMA_EPI && EPI == EPI_GLU_BWD;
      [[maybe_unused]] uint4 gv[2][NP], uv[2][NP];
      auto glu_fetch = [&](int step) {
        if constexpr (kGluRegs) {
          const int col0 = t.n0 + half * (BN / 2) + (step >> 1) * CW;
          const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(p.aux) +
                                     static_cast<long long>(row0 + 16 * (step & 1)) * p.ld2 + col0;
#pragma unroll
          for (int s2 = 0; s2 < 2; ++s2) {
            epi_pieces<NP>(src + 8LL * s2 * p.ld2, p.ld2, p.I - col0, lane, gv[s2]);
            epi_pieces<NP>(src + 8LL * s2 * p.ld2 + p.I, p.ld2, p.I - col0, lane, uv[s2]);
          }
        }
      };
      glu_fetch(0);
      if (!mbar_wait(bar_tfull + 8 * buf, (it >> 1) & 1, abort_flag, ST_WAIT_EPILOGUE)) break;
      __syncwarp();
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * BN;
      const bool have_acc = t.nkb > 0;

      if constexpr (TMA_EPI) {
        // results are packed to bf16, staged per warp as 32 rows x 64 columns and written by TMA
        // stores (which clip at the tensor's bounds, so no row or column masks are needed)
        uint8_t* sbuf = bufG;   // this warp's staging box
        const int grp = (p.sched == SCHED_GROUPED_K || (CONV && p.conv_taps > 0)) ? t.g : 0;
        if constexpr (EPI == EPI_STORE || EPI == EPI_AXPBY || EPI == EPI_STORE_SYM) {
          constexpr int W = BN / 2;
          // push mode: this lane's output row goes to a slot of another GPU's (or this GPU's) receive buffer
          uint8_t* push_dst = nullptr;
          if (p.push_rank != nullptr) {
            const int rk = p.push_rank[row];
            if (rk >= 0)
              push_dst = reinterpret_cast<uint8_t*>(p.push_base[rk]) + static_cast<long long>(p.push_slot[row]) * p.N * 2;
          }
          const int ax_drow = (EPI == EPI_AXPBY) ? static_cast<int>(row) - p.poffs[t.g] : 0;   // row inside its group
#pragma unroll 1
          for (int c = half * W; c < (half + 1) * W; c += 64) {
            if (t.n0 + c >= p.N) break;
            uint32_t pk[32];
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
              uint32_t r[32];
              if (have_acc) {
                tmem_ld32(taddr + c + 32 * sub, r);
                tmem_ld_wait();
              } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = 0u;
              }
              if constexpr (EPI == EPI_AXPBY) {
                // r = alpha * acc + beta * C[row, columns] (+ diag on the group's own diagonal); the lane reads the
                // 64 bytes of its row of C that lie under this sub-chunk
                const int col0 = t.n0 + c + 32 * sub;
                const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.aux) +
                                                                  row * p.ldd + col0);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                  const uint4 cv = src[v];
                  const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                  for (int h = 0; h < 4; ++h) {
                    const float2 cf = unpack_bf16x2(cw[h]);
                    const int i = 8 * v + 2 * h;
                    float v0 = p.ax_alpha * __uint_as_float(r[i]) + p.ax_beta * cf.x;
                    float v1 = p.ax_alpha * __uint_as_float(r[i + 1]) + p.ax_beta * cf.y;
                    if (col0 + i == ax_drow) v0 += p.ax_diag;
                    if (col0 + i + 1 == ax_drow) v1 += p.ax_diag;
                    r[i] = __float_as_uint(v0);
                    r[i + 1] = __float_as_uint(v1);
                  }
                }
              }
#pragma unroll
              for (int i = 0; i < 16; ++i)
                pk[16 * sub + i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            }
            if (p.push_rank != nullptr) {
              // each lane stages its own 128-byte row piece (unswizzled) and sends it with one bulk copy
              bulk_wait_read_all();   // this lane's previous copy has read the piece
              uint8_t* mine = sbuf + lane * 128;
#pragma unroll
              for (int j = 0; j < 8; ++j)
                *reinterpret_cast<uint4*>(mine + 16 * j) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
              fence_proxy_async_smem();
              if (push_dst != nullptr) {
                const int left = (p.N - (t.n0 + c)) * 2;
                bulk_store_1d(push_dst + static_cast<long long>(t.n0 + c) * 2, smem_u32(mine), left < 128 ? left : 128);
              }
              bulk_commit_group();
            } else {
              staging_free(lane);
              stage_row(sbuf, lane, pk);
              store_box(&tmD, sbuf, lane, t.n0 + c, row0, grp);
              if constexpr (EPI == EPI_AXPBY || EPI == EPI_STORE_SYM) if (p.sym_mirror) {
                // symmetric result: the chunk (32 rows x 64 columns) of a tile right of the diagonal tile is also
                // the transpose of a chunk nobody computes.  Stage it as 64 rows x 32 columns (unswizzled rows of
                // 64 bytes; lane l owns column l) and store it through the second map.
                const int lrow0 = row0 - t.g * p.sym_rows;          // this warp's first row inside its group
                if ((t.n0 + c) / B200MOE_TILE_M > lrow0 / B200MOE_TILE_M) {
                  staging_free(lane);                               // the store above has read the box
#pragma unroll
                  for (int m = 0; m < 32; ++m) {
                    *reinterpret_cast<uint16_t*>(sbuf + (2 * m) * 64 + lane * 2) = static_cast<uint16_t>(pk[m] & 0xffffu);
                    *reinterpret_cast<uint16_t*>(sbuf + (2 * m + 1) * 64 + lane * 2) = static_cast<uint16_t>(pk[m] >> 16);
                  }
                  store_box(&tmD2, sbuf, lane, lrow0, t.g * p.sym_rows + t.n0 + c, 0);
                }
              }
            }
          }
        } else if constexpr (EPI == EPI_SWIGLU) {
          // accumulator columns [0,BN/2) = gate, [BN/2,BN) = up for I-columns [n0, n0+BN/2)
          const int c = half * (BN / 4);
          if (t.n0 + c < p.I) {
            uint32_t og[32], ou[32], oh[32];
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
              uint32_t g[32], u[32];
              tmem_ld32(taddr + c + 32 * sub, g);
              tmem_ld32(taddr + BN / 2 + c + 32 * sub, u);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                og[16 * sub + i] = pack_bf16x2(__uint_as_float(g[2 * i]), __uint_as_float(g[2 * i + 1]));
                ou[16 * sub + i] = pack_bf16x2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
              }
              glu_fwd_pairs_by_code<POLY>(act_code, og + 16 * sub, ou + 16 * sub, oh + 16 * sub, 16);
            }
            staging_free(lane);
            stage_row(sbuf, lane, og);
            store_box(&tmD, sbuf, lane, t.n0 + c, row0, 0);    // gate half of gate_up
            staging_free(lane);
            stage_row(sbuf, lane, ou);
            store_box(&tmD, sbuf, lane, t.n0 + c, row0, 1);    // up half
            staging_free(lane);
            stage_row(sbuf, lane, oh);
            store_box(&tmD2, sbuf, lane, t.n0 + c, row0, 0);   // inter
          }
        } else {  // EPI_GLU_BWD: accumulator = grad_inter columns [n0, n0+BN); this warp: 128 of them
          constexpr int W = BN / 2;
#pragma unroll 1
          for (int sub = 0; sub < W / 32; ++sub) {
            const int col = glu_col0 + 32 * sub;
            if (col >= p.I) break;                       // warp-uniform
            const int set = sub & 1;
            uint8_t* bG = ebuf + set * 2 * kGluBoxBytes;
            uint8_t* bU = bG + kGluBoxBytes;
            uint32_t r[32];
            tmem_ld32(taddr + half * W + 32 * sub, r);
            if (!mbar_wait(ebar + 8 * set, (epi_phase >> set) & 1u, abort_flag, ST_WAIT_EPILOGUE)) break;
            epi_phase ^= 1u << set;
            uint4 g4[4], u4[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {              // this lane's row: 64 bytes, 64-byte swizzle
              const int off = lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4);
              g4[v] = *reinterpret_cast<const uint4*>(bG + off);
              u4[v] = *reinterpret_cast<const uint4*>(bU + off);
            }
            tmem_ld_wait();
            uint32_t og[16], ou[16];
            glu_bwd32<POLY>(r, g4, u4, og, ou, act_code);
#pragma unroll
            for (int v = 0; v < 4; ++v) {              // results replace the inputs in place
              const int off = lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4);
              *reinterpret_cast<uint4*>(bG + off) = make_uint4(og[4 * v], og[4 * v + 1], og[4 * v + 2], og[4 * v + 3]);
              *reinterpret_cast<uint4*>(bU + off) = make_uint4(ou[4 * v], ou[4 * v + 1], ou[4 * v + 2], ou[4 * v + 3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&tmD, smem_u32(bG), col, row0, 0);   // grad_gate
              tma_store_3d(&tmD, smem_u32(bU), col, row0, 1);   // grad_up
              bulk_commit_group();
            }
            // as soon as that store has read its boxes (a few hundred ns), they are reloaded with the sub-chunk
            // after the next one, which then has a whole sub-chunk of arithmetic to arrive
            if (sub + 2 < W / 32 && glu_col0 + 32 * (sub + 2) < p.I) {
              staging_free(lane);
              glu_load(sub + 2);
            }
          }
        }
      } else {
        // Single-CTA tiles up to 128 wide, and fp32 partial sums: from tensor memory through registers.  16 rows x 64 (or 32) columns at a
        // time are read as 8 x 8 blocks; among the four threads that hold a row's blocks a 4 x 4 exchange of packed words gives each one
        // block's 16 bytes, and a second one between neighbouring rows lets a warp read or write 128 contiguous bytes of 4 rows per
        // instruction.  (Each lane writing 16-byte pieces of its own row: 512 tokens of H 256, I 512, 8 experts: gate/up 7.4 us against
        // 6.2, GLU backward 12.2 against 8.7, the four other products on such tiles 27.1 against 25.4; fp32 partial sums of 256 x 2048 26.0
        // against 23.1.)
        const uint32_t lower = taddr + (16u << 16);      // rows 16 ... of the warp
        if constexpr (EPI == EPI_STORE || EPI == EPI_STORE_F32) {
          constexpr int W = BN / 2;                     // columns per warp
          const bool conv_rows = CONV && p.conv_taps > 0 && p.sched == SCHED_DENSE;   // rows are positions of batch t.g
          const int rows_end = (p.sched == SCHED_GROUPED_M) ? 0x7fffffff : (conv_rows ? p.conv_S : p.M);
          const long long base = ((p.sched == SCHED_GROUPED_K || conv_rows) ? t.g * p.d_group_stride : 0) +
                                 static_cast<long long>(row0) * p.ldd + t.n0 + half * W;
          const int live = min(W, p.N - t.n0 - half * W);                             // columns of this warp
#pragma unroll 1
          for (int c = 0; c < live; c += CW) {
            uint32_t r[2][NP][16];
            epi_load<NP>(taddr + half * W + c, have_acc, r[0]);
            epi_load<NP>(lower + half * W + c, have_acc, r[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int rows = rows_end - row0 - 8 * i;
              if constexpr (EPI == EPI_STORE_F32) {
                float* d = reinterpret_cast<float*>(p.D) + base + static_cast<long long>(8 * i + (lane >> 2)) * p.ldd + c + 2 * (lane & 3);
#pragma unroll
                for (int b = 0; b < 4 * NP; ++b)
                  if ((lane >> 2) < rows && c + 8 * b < live)
                    *reinterpret_cast<uint2*>(d + 8 * b) = make_uint2(r[i >> 1][b / 4][4 * (b % 4) + 2 * (i & 1)], r[i >> 1][b / 4][4 * (b % 4) + 2 * (i & 1) + 1]);
              } else {
                uint32_t w[NP][4];
#pragma unroll
                for (int j = 0; j < NP; ++j) epi_pack(r[i >> 1][j], i & 1, w[j]);
                epi_put<NP>(reinterpret_cast<__nv_bfloat16*>(p.D) + base + static_cast<long long>(8 * i) * p.ldd + c, p.ldd, rows, live - c, lane, w);
              }
            }
          }
        } else if constexpr (EPI == EPI_SWIGLU) {
          // accumulator columns [0,BN/2) = gate, [BN/2,BN) = up for I-columns [n0, n0+BN/2)
          const int I = p.I, c = half * (BN / 4), col0 = t.n0 + c;
          if (col0 < I) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              uint32_t g[NP][16], u[NP][16];
              epi_load<NP>((h ? lower : taddr) + c, true, g);
              epi_load<NP>((h ? lower : taddr) + BN / 2 + c, true, u);
              tmem_ld_wait();
#pragma unroll
              for (int s2 = 0; s2 < 2; ++s2) {
                const long long r8 = row0 + 16 * h + 8 * s2;
                uint32_t gw[NP][4], uw[NP][4], hw[NP][4];
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                  epi_pack(g[i], s2, gw[i]);
                  epi_pack(u[i], s2, uw[i]);
                  glu_fwd_pairs_by_code<POLY>(act_code, gw[i], uw[i], hw[i], 4);
                }
                __nv_bfloat16* gu = reinterpret_cast<__nv_bfloat16*>(p.D) + r8 * p.ld2 + col0;
                epi_put<NP>(gu, p.ld2, 8, I - col0, lane, gw);
                epi_put<NP>(gu + I, p.ld2, 8, I - col0, lane, uw);
                epi_put<NP>(reinterpret_cast<__nv_bfloat16*>(p.aux) + r8 * p.ldi + col0, p.ldi, 8, I - col0, lane, hw);
              }
            }
          }
        } else {  // EPI_GLU_BWD: accumulator = grad_inter columns [n0, n0+BN)
          constexpr int W = BN / 2;
          const int I = p.I;
#pragma unroll 1
          for (int step = 0; step < W / CW * 2; ++step) {
            const int c = half * W + (step >> 1) * CW, col0 = t.n0 + c;
            if (col0 >= I) break;
            uint32_t gw[2][NP][4], uw[2][NP][4], r[NP][16];
#pragma unroll
            for (int s2 = 0; s2 < 2; ++s2) {
              epi_words<NP>(gv[s2], lane, gw[s2]);
              epi_words<NP>(uv[s2], lane, uw[s2]);
            }
            if (step + 1 < W / CW * 2) glu_fetch(step + 1);
            epi_load<NP>(((step & 1) ? lower : taddr) + c, true, r);
            tmem_ld_wait();
#pragma unroll
            for (int s2 = 0; s2 < 2; ++s2) {
#pragma unroll
              for (int i = 0; i < NP; ++i) {
                uint32_t iw[4];
                epi_pack(r[i], s2, iw);                         // rounded to bf16: the reference materialises grad_inter in bf16
                glu_bwd_pairs<POLY>(act_code, iw, gw[s2][i], uw[s2][i]);      // now grad_gate, grad_up
              }
              __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + static_cast<long long>(row0 + 16 * (step & 1) + 8 * s2) * p.ld2 + col0;
              epi_put<NP>(d, p.ld2, 8, I - col0, lane, gw[s2]);
              epi_put<NP>(d + I, p.ld2, 8, I - col0, lane, uw[s2]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (CTAS == 2) mbar_arrive_cluster(tempty_leader + 8 * buf);
        else mbar_arrive(bar_tempty + 8 * buf);
      }
    }
    if constexpr (TMA_EPI) {
      if (lane == 0 || p.push_rank != nullptr) bulk_wait_all();   // every bulk store of this warp (push mode: of this lane) has completed
    }
  }

  // ------------------------------------------------------------------ tear-down
  tc_fence_before();
  __syncthreads();
  if constexpr (CTAS == 2) {   // nobody leaves while the peer may still touch it
    __syncwarp();
    cluster_sync_all();
  }
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_flag);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if constexpr (CTAS == 2) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
    else tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------- host side
template <int BN, int EPI, int CTAS, bool POLY = false>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmD, const CUtensorMap& tmD2,
                  const GemmParams& p, int max_tiles, cudaStream_t stream) {
  using C = Cfg<BN, CTAS, epi_warp_bytes<BN, EPI>()>;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_kernel<BN, EPI, CTAS, POLY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    C::SMEM_BYTES);
  });
  if (attr_err != cudaSuccess) return cuda_fail(attr_err, "cudaFuncSetAttribute(max dynamic smem)");
  int units = gemm_cta_budget() / CTAS;  // CTAs, or CTA pairs
  if (max_tiles > 0 && max_tiles < units) units = max_tiles;
  if (units < 1) units = 1;
  B200_CUDA(launch_chained(gemm_kernel<BN, EPI, CTAS, POLY>, units * CTAS, gemm_threads(CTAS), C::SMEM_BYTES, stream, CTAS, tmA, tmB, tmD, tmD2, p));
  return 0;
}

// Pair (2-CTA) tiles are used for the grouped schedules with 256-wide tiles.  Setting the
// environment variable B200MOE_FORCE_1CTA=1 keeps every launch on single-CTA tiles (A/B measurements).
static bool pairs_enabled() {
  static int v = -1;
  static std::once_flag once;
  std::call_once(once, [] {
    const char* e = getenv("B200MOE_FORCE_1CTA");
    v = (e != nullptr && e[0] == '1') ? 0 : 1;
  });
  return v == 1;
}

// Operand description used by the host-side dispatcher.
struct Operand {
  const void* ptr;
  int mn_major;         // 0: (rows, K) row-major;  1: (K, rows) row-major
  long long rows;       // M (for A) or N (for B)
  long long k;          // reduction extent visible in this tensor
  long long ld;         // elements between consecutive rows of the stored matrix
  long long groups;     // stacked matrices (experts), 1 if none
  long long group_stride;
};

static int encode_operand(CUtensorMap* tm, const Operand& o, int tile_rows) {
  if (!o.mn_major)  // dims {K, rows, groups}, box {64, tile_rows}
    return make_map(tm, o.ptr, o.k, o.rows, o.groups, o.ld, o.group_stride, BK, tile_rows);
  // dims {rows(mn), K, groups}, box {64 mn, 64 k}
  return make_map(tm, o.ptr, o.rows, o.k, o.groups, o.ld, o.group_stride, 64, BK);
}

static int pick_bn(long long n) {
  if (n <= 64) return 64;
  if (n % 256 == 0 || n > 1024) {
    // prefer the wide tile unless it wastes more than 1/8 of the last tile
    long long waste256 = ((n + 255) / 256) * 256 - n;
    if (waste256 * 8 <= n) return 256;
  }
  return 128;
}

// Tile width of the grouped products: pair tiles (256 x 256 on two SMs), or single-CTA tiles 128 wide (`narrow`: the least
// the epilogue is built for).  m_tiles = 256-row tiles, m_tiles1 = 128-row tiles over all groups.  Waves of tiles over the
// machine decide: a wave of 128 x 128 tiles takes about 0.8 of a wave of pair tiles for half of its work per SM (0.9 with a
// long reduction, 0.6 with a short one), so small products, whose pair tiles leave most SMs idle, run faster on it.
// us, pair against single-CTA tiles: 8 experts x 500 rows, 264 x 136: down 9.5 / 6.6, weight gradients 14.8 / 8.5 and
// 14.3 / 8.5; 32 experts x 375 rows, 1032 x 680: 38 / 49, 54 / 80, 36 / 55; 16 experts x 1000 rows, 1800 x 968: 72 / 107,
// 104 / 176, 62 / 99.
static int pick_bn_grouped(long long n, int narrow, long long m_tiles, long long m_tiles1, int cols_per_bn = 1) {
  if (n * cols_per_bn <= 64) return narrow;
  if (!pairs_enabled()) return std::max(pick_bn(n), narrow);
  const long long units = gemm_cta_budget();
  const long long pair_waves = ceil_div(m_tiles * ceil_div(n * cols_per_bn, 256), units / 2);
  const long long cta_waves = ceil_div(m_tiles1 * ceil_div(n * cols_per_bn, 128), units);
  return 10 * pair_waves <= 8 * cta_waves ? 256 : 128;
}
// the same over the padded rows of a routing decision, of which each group's last tile is taken to be half full
static int pick_bn_rows(long long n, long long rows_cap, int E, int cols_per_bn = 1) {
  const long long t = std::max<long long>(1, rows_cap / B200MOE_TILE_M - E / 2);
  return pick_bn_grouped(n, 128, t, 2 * t, cols_per_bn);
}

// d1 / d2 describe the bf16 outputs as {columns, rows, groups} tensors for the TMA-store epilogue
// (d2 = the SwiGLU `inter` output); they are ignored by the kernels that store directly.
template <int EPI, bool POLY = false>
static int dispatch_bn(int bn, const Operand& A, const Operand& B, const Operand* d1, const Operand* d2,
                       GemmParams& p, int max_tiles, cudaStream_t stream) {
  const bool pair = (bn == 256) && (p.sched != SCHED_DENSE) && pairs_enabled();
  CUtensorMap tmA, tmB, tmD, tmD2;
  int rc = encode_operand(&tmA, A, BM);
  if (rc) return rc;
  // rows of B one TMA box brings in: half a tile for SwiGLU (gate and up halves) and for pairs
  const int b_rows = (EPI == EPI_SWIGLU || pair) ? bn / 2 : bn;
  rc = encode_operand(&tmB, B, b_rows);
  if (rc) return rc;
  tmD = tmA;
  tmD2 = tmA;
  if (bn == 256 && EPI != EPI_STORE_F32 && p.push_rank == nullptr) {
    if (d1 == nullptr) {
      set_error("internal: output description missing");
      return B200MOE_E_UNSUPPORTED;
    }
    if (EPI == EPI_GLU_BWD) {   // boxes {32 columns, 32 rows}, 64-byte swizzle, for the in-place epilogue
      if (d2 == nullptr) {
        set_error("internal: saved gate_up description missing");
        return B200MOE_E_UNSUPPORTED;
      }
      rc = make_map(&tmD, d1->ptr, d1->k, d1->rows, d1->groups, d1->ld, d1->group_stride, 32, 32, 2, 64);
      if (rc) return rc;
      rc = make_map(&tmD2, d2->ptr, d2->k, d2->rows, d2->groups, d2->ld, d2->group_stride, 32, 32, 2, 64);
      if (rc) return rc;
    } else {
      rc = encode_operand(&tmD, *d1, 32);   // box {64 columns, 32 rows}
      if (rc) return rc;
      if (d2 != nullptr) {
        rc = encode_operand(&tmD2, *d2, 32);
        if (rc) return rc;
      } else if (p.sym_mirror) {            // the same output through boxes {32 columns, 64 rows}, no swizzle
        rc = make_map(&tmD2, d1->ptr, d1->k, d1->rows, d1->groups, d1->ld, d1->group_stride, 32, 64, 2, 0);
        if (rc) return rc;
      }
    }
  }
  if (pair) return launch<256, EPI, 2, POLY>(tmA, tmB, tmD, tmD2, p, max_tiles > 0 ? (max_tiles + 1) / 2 : 0, stream);
  if constexpr (EPI == EPI_AXPBY || EPI == EPI_STORE_SYM) {   // built for the 256-wide TMA-store epilogue only
    if (bn == 256) return launch<256, EPI, 1>(tmA, tmB, tmD, tmD2, p, max_tiles, stream);
    set_error("tile width %d not built for this epilogue", bn);
    return B200MOE_E_UNSUPPORTED;
  } else
  switch (bn) {
    case 256: return launch<256, EPI, 1, POLY>(tmA, tmB, tmD, tmD2, p, max_tiles, stream);
    case 128: return launch<128, EPI, 1, POLY>(tmA, tmB, tmD, tmD2, p, max_tiles, stream);
    default:
      if constexpr (EPI == EPI_STORE || EPI == EPI_STORE_F32)
        return launch<64, EPI, 1, POLY>(tmA, tmB, tmD, tmD2, p, max_tiles, stream);
      set_error("tile width %d not built for this epilogue", bn);
      return B200MOE_E_UNSUPPORTED;
  }
}


static int check_grouped(const char* who, const void* a, const void* b, const void* c, const int32_t* tile_expert,
                         const int32_t* poffs, int64_t rows_cap, int E, int64_t H, int64_t I) {
  B200_CHECK_ARG(a && b && c && poffs, B200MOE_E_NULL, "%s: null pointer", who);
  (void)tile_expert;
  B200_CHECK_ARG(E >= 1 && E <= 65535, B200MOE_E_BAD_SHAPE, "%s: E = %d out of range", who, E);
  B200_CHECK_ARG(rows_cap > 0 && rows_cap % B200MOE_TILE_M == 0 && rows_cap < (1LL << 31), B200MOE_E_BAD_SHAPE,
                 "%s: rows_cap = %lld must be a positive multiple of %d", who, (long long)rows_cap, B200MOE_TILE_M);
  B200_CHECK_ARG(H > 0 && H % 8 == 0 && I > 0 && I % 8 == 0, B200MOE_E_BAD_SHAPE,
                 "%s: H = %lld and I = %lld must be positive multiples of 8", who, (long long)H, (long long)I);
  B200_CHECK_ARG(2 * E * I < (1LL << 31) && E * H < (1LL << 31), B200MOE_E_BAD_SHAPE, "%s: weight stack too tall", who);
  return 0;
}

// ---- products of equal groups of padded rows (the optimizer's iteration; linear_t also the layer's).  n_live / k_live: columns
// that are computed and the part of the reduction that is read, multiples of 64 that cover what is not padding (n_live, k_live =
// the whole extent otherwise).  What lies past them is neither read nor, where a whole 64-column chunk is padding, written.
int expert_gram(const void* x, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t K, int mirror,
                int64_t n_live, void* out, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(E >= 1 && rows_cap % E == 0, B200MOE_E_BAD_SHAPE, "expert_gram: %lld rows do not split into %d equal groups",
                 (long long)rows_cap, E);
  const int64_t R = rows_cap / E;
  int rc = check_grouped("expert_gram", x, x, out, tile_expert, poffs, rows_cap, E, R, K);
  if (rc) return rc;
  B200_CHECK_ARG(tile_expert, B200MOE_E_NULL, "expert_gram: null pointer");
  B200_CHECK_ARG(R % 256 == 0, B200MOE_E_BAD_SHAPE, "expert_gram: %lld rows per group must be a multiple of 256", (long long)R);
  B200_CHECK_ARG(aligned16(out), B200MOE_E_ALIGN, "expert_gram: output not aligned");
  Operand oa{x, 0, rows_cap, K, K, 1, rows_cap * K};
  Operand ob{x, 0, R, K, K, E, R * K};
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.N = (int)n_live; p.K = (int)K; p.num_groups = E; p.sym_rows = (int)R; p.sym_mirror = mirror ? 1 : 0;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = out; p.ldd = R; p.status = status;
  Operand d{out, 0, rows_cap, R, R, 1, rows_cap * R};
  return dispatch_bn<EPI_STORE_SYM>(256, oa, ob, &d, nullptr, p, 0, (cudaStream_t)stream);
}

int expert_linear_axpby(const void* a, const void* w, const void* c, float alpha, float beta, float diag, int symmetric,
                        const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t N, int64_t K,
                        int64_t n_live, int64_t k_live, void* out, int32_t* status, b200moe_stream_t stream) {
  int rc = check_grouped("expert_linear_axpby", a, w, out, tile_expert, poffs, rows_cap, E, N, K);
  if (rc) return rc;
  B200_CHECK_ARG(tile_expert && c, B200MOE_E_NULL, "expert_linear_axpby: null pointer");
  B200_CHECK_ARG(N % 256 == 0, B200MOE_E_BAD_SHAPE, "expert_linear_axpby: N = %lld must be a multiple of 256", (long long)N);
  B200_CHECK_ARG(aligned16(out) && aligned16(c), B200MOE_E_ALIGN, "expert_linear_axpby: pointers must be 16-byte aligned");
  Operand oa{a, 0, rows_cap, k_live, K, 1, rows_cap * K};
  Operand ob{w, 0, N, k_live, K, E, N * K};   // W (E, N, K): rows = output columns
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.N = (int)n_live; p.K = (int)k_live; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = out; p.ldd = N; p.status = status;
  p.aux = const_cast<void*>(c); p.ax_alpha = alpha; p.ax_beta = beta; p.ax_diag = diag;
  if (symmetric) {
    B200_CHECK_ARG(rows_cap == (int64_t)E * N, B200MOE_E_BAD_SHAPE,
                   "expert_linear_axpby: a symmetric result needs %d equal groups of N = %lld rows", E, (long long)N);
    p.sym_rows = (int)N;
    p.sym_mirror = symmetric > 1 ? 1 : 0;
  }
  Operand d{out, 0, rows_cap, N, N, 1, rows_cap * N};
  return dispatch_bn<EPI_AXPBY>(256, oa, ob, &d, nullptr, p, 0, (cudaStream_t)stream);
}

int expert_linear_t(const void* a, int64_t lda, const void* w, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E,
                    int64_t K, int64_t N, int64_t k_live, void* out, int64_t ldo, int32_t* status, b200moe_stream_t stream) {
  int rc = check_grouped("expert_linear_t", a, w, out, tile_expert, poffs, rows_cap, E, N, K);
  if (rc) return rc;
  B200_CHECK_ARG(tile_expert, B200MOE_E_NULL, "expert_linear_t: null pointer");
  B200_CHECK_ARG(aligned16(out), B200MOE_E_ALIGN, "expert_linear_t: output not aligned");
  Operand oa{a, 0, rows_cap, k_live, lda, 1, rows_cap * lda};
  Operand ob{w, 1, N, k_live, N, E, K * N};   // W[e] stored (K, N): MN-major
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.b_mn = 1; p.N = (int)N; p.K = (int)k_live; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = out; p.ldd = ldo; p.status = status;
  Operand d{out, 0, rows_cap, N, ldo, 1, rows_cap * ldo};
  return dispatch_bn<EPI_STORE>(pick_bn_rows(N, rows_cap, E), oa, ob, &d, nullptr, p, 0, (cudaStream_t)stream);
}

// row window of a grouped-M launch: (0, 0) = every row, else tile-aligned 0 <= row_lo < row_hi <= rows_cap
static int check_row_window(const char* who, int64_t rows_cap, int64_t row_lo, int64_t row_hi) {
  if (row_lo == 0 && row_hi == 0) return 0;
  B200_CHECK_ARG(row_lo >= 0 && row_lo < row_hi && row_hi <= rows_cap && row_lo % B200MOE_TILE_M == 0 &&
                     row_hi % B200MOE_TILE_M == 0,
                 B200MOE_E_BAD_SHAPE, "%s: row window [%lld, %lld) must be tile-aligned and inside %lld rows", who,
                 (long long)row_lo, (long long)row_hi, (long long)rows_cap);
  return 0;
}

int expert_gate_up(const void* x_s, int64_t ldh, const void* gate_up_proj, const int32_t* act_codes, const int32_t* tile_expert,
                   const int32_t* poffs, int64_t rows_cap, int64_t row_lo, int64_t row_hi, int E, int64_t H, int64_t I, void* gate_up, int64_t ld2,
                   void* inter, int64_t ldi, int32_t* status, b200moe_stream_t stream) {
  int rc = check_grouped("expert_gate_up_swiglu", x_s, gate_up_proj, gate_up, tile_expert, poffs, rows_cap, E, H, I);
  if (rc) return rc;
  rc = check_row_window("expert_gate_up_swiglu", rows_cap, row_lo, row_hi);
  if (rc) return rc;
  B200_CHECK_ARG(inter && tile_expert, B200MOE_E_NULL, "expert_gate_up_swiglu: null pointer");
  B200_CHECK_ARG(aligned16(gate_up) && aligned16(inter), B200MOE_E_ALIGN, "expert_gate_up_swiglu: outputs not aligned");
  Operand a{x_s, 0, rows_cap, H, ldh, 1, rows_cap * ldh};
  // W_gu (E, 2I, H) seen as dims {H, I, 2E}: group 2e = gate rows of expert e, 2e+1 = up rows
  Operand b{gate_up_proj, 0, I, H, H, 2LL * E, I * H};
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.N = (int)I; p.K = (int)H; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = gate_up; p.aux = inter; p.I = (int)I; p.ld2 = ld2; p.ldi = ldi;
  p.status = status;
  p.row_lo = (int)row_lo; p.row_hi = (int)row_hi;
  const int bn = pick_bn_rows(I, rows_cap, E, 2);   // tile covers bn/2 intermediate columns
  Operand d1{gate_up, 0, rows_cap, I, ld2, 2, I};         // {I, rows, 2}: group 0 = gate half, 1 = up half
  Operand d2{inter, 0, rows_cap, I, ldi, 1, rows_cap * ldi};
  p.act_codes = act_codes;
  if (act_codes != nullptr) return dispatch_bn<EPI_SWIGLU, true>(bn, a, b, &d1, &d2, p, 0, (cudaStream_t)stream);
  return dispatch_bn<EPI_SWIGLU>(bn, a, b, &d1, &d2, p, 0, (cudaStream_t)stream);
}

int expert_down_dgrad(const void* grad_eo, int64_t ldh, const void* down_proj, const void* gate_up, int64_t ld2, const int32_t* act_codes,
                      const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int64_t row_lo, int64_t row_hi, int E,
                      int64_t H, int64_t I, void* grad_gate_up, int32_t* status, b200moe_stream_t stream) {
  int rc = check_grouped("expert_down_dgrad_glu", grad_eo, down_proj, grad_gate_up, tile_expert, poffs, rows_cap, E, H, I);
  if (rc) return rc;
  rc = check_row_window("expert_down_dgrad_glu", rows_cap, row_lo, row_hi);
  if (rc) return rc;
  B200_CHECK_ARG(gate_up && tile_expert, B200MOE_E_NULL, "expert_down_dgrad_glu: null pointer");
  B200_CHECK_ARG(aligned16(grad_gate_up) && aligned16(gate_up), B200MOE_E_ALIGN, "expert_down_dgrad_glu: not aligned");
  Operand a{grad_eo, 0, rows_cap, H, ldh, 1, rows_cap * ldh};
  Operand b{down_proj, 1, I, H, I, E, H * I};   // W_d[e] stored (K=H, N=I): MN-major
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.b_mn = 1; p.N = (int)I; p.K = (int)H; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = grad_gate_up; p.aux = const_cast<void*>(gate_up);
  p.I = (int)I; p.ld2 = ld2; p.status = status;
  p.row_lo = (int)row_lo; p.row_hi = (int)row_hi;
  const int bn = pick_bn_rows(I, rows_cap, E);
  Operand d{grad_gate_up, 0, rows_cap, I, ld2, 2, I};     // {I, rows, 2}: grad_gate half, grad_up half
  Operand d2{gate_up, 0, rows_cap, I, ld2, 2, I};         // the saved forward gate_up, same view (input)
  p.act_codes = act_codes;
  if (act_codes != nullptr) return dispatch_bn<EPI_GLU_BWD, true>(bn, a, b, &d, &d2, p, 0, (cudaStream_t)stream);
  return dispatch_bn<EPI_GLU_BWD>(bn, a, b, &d, &d2, p, 0, (cudaStream_t)stream);
}

int expert_linear(const void* a, int64_t lda, const void* w, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E, int64_t N,
                  int64_t K, void* out, int64_t ldo, int32_t* status, b200moe_stream_t stream) {
  int rc = check_grouped("expert_linear", a, w, out, tile_expert, poffs, rows_cap, E, N, K);
  if (rc) return rc;
  B200_CHECK_ARG(tile_expert, B200MOE_E_NULL, "expert_linear: null pointer");
  B200_CHECK_ARG(aligned16(out), B200MOE_E_ALIGN, "expert_linear: output not aligned");
  Operand oa{a, 0, rows_cap, K, lda, 1, rows_cap * lda};
  Operand ob{w, 0, N, K, K, E, N * K};   // W (E, N, K): rows = output columns
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.N = (int)N; p.K = (int)K; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = out; p.ldd = ldo; p.status = status;
  Operand d{out, 0, rows_cap, N, ldo, 1, rows_cap * ldo};
  return dispatch_bn<EPI_STORE>(pick_bn_rows(N, rows_cap, E), oa, ob, &d, nullptr, p, 0, (cudaStream_t)stream);
}

int expert_wgrad(const void* A, int64_t lda, const void* B, int64_t ldb, const int32_t* poffs, const int32_t* counts, int64_t rows_cap, int E,
                 int64_t Na, int64_t Nb, void* out, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(A && B && poffs && out, B200MOE_E_NULL, "expert_wgrad: null pointer");
  B200_CHECK_ARG(E >= 1, B200MOE_E_BAD_SHAPE, "expert_wgrad: E = %d", E);
  B200_CHECK_ARG(rows_cap > 0 && rows_cap % B200MOE_TILE_M == 0 && rows_cap < (1LL << 31), B200MOE_E_BAD_SHAPE,
                 "expert_wgrad: rows_cap = %lld must be a positive multiple of %d", (long long)rows_cap, B200MOE_TILE_M);
  CHECK_DIM8(Na); CHECK_DIM8(Nb); CHECK_I32(Na); CHECK_I32(Nb);
  B200_CHECK_ARG(aligned16(out), B200MOE_E_ALIGN, "expert_wgrad: output not aligned");
  Operand a{A, 1, Na, rows_cap, lda, 1, rows_cap * lda};
  Operand b{B, 1, Nb, rows_cap, ldb, 1, rows_cap * ldb};
  GemmParams p{};
  p.sched = SCHED_GROUPED_K; p.a_mn = 1; p.b_mn = 1; p.M = (int)Na; p.N = (int)Nb; p.K = (int)rows_cap;
  p.num_groups = E; p.poffs = poffs; p.counts = counts; p.D = out; p.ldd = Nb; p.d_group_stride = Na * Nb;
  p.status = status;
  const int bn = pick_bn_grouped(Nb, 64, E * ceil_div(Na, 256), E * ceil_div(Na, BM));
  Operand d{out, 0, Na, Nb, Nb, E, Na * Nb};
  const int tiles = (int)std::min<long long>(1 << 30, E * ceil_div(Na, BM) * ceil_div(Nb, bn));
  return dispatch_bn<EPI_STORE>(bn, a, b, &d, nullptr, p, tiles, (cudaStream_t)stream);
}

}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_gemm_nt(const void* A, const void* B, void* D, int64_t M, int64_t N, int64_t K, int32_t* status,
                    b200moe_stream_t stream) {
  B200_CHECK_ARG(A && B && D, B200MOE_E_NULL, "gemm_nt: null pointer");
  CHECK_DIM8(N); CHECK_DIM8(K); CHECK_I32(M); CHECK_I32(N); CHECK_I32(K);
  if (M == 0) return 0;
  B200_CHECK_ARG(aligned16(D), B200MOE_E_ALIGN, "gemm_nt: D not 16-byte aligned");
  Operand a{A, 0, M, K, K, 1, M * K};
  Operand b{B, 0, N, K, K, 1, N * K};
  GemmParams p{};
  p.sched = SCHED_DENSE; p.M = (int)M; p.N = (int)N; p.K = (int)K; p.num_groups = 1;
  p.D = D; p.ldd = N; p.status = status;
  const int bn = pick_bn(N);
  Operand d{D, 0, M, N, N, 1, M * N};
  return dispatch_bn<EPI_STORE>(bn, a, b, &d, nullptr, p, (int)(ceil_div(M, BM) * ceil_div(N, bn)), (cudaStream_t)stream);
}

int b200moe_gemm_nn(const void* A, const void* B, void* D, int64_t M, int64_t N, int64_t K, int32_t* status,
                    b200moe_stream_t stream) {
  B200_CHECK_ARG(A && B && D, B200MOE_E_NULL, "gemm_nn: null pointer");
  CHECK_DIM8(N); CHECK_DIM8(K); CHECK_I32(M); CHECK_I32(N); CHECK_I32(K);
  if (M == 0) return 0;
  B200_CHECK_ARG(aligned16(D), B200MOE_E_ALIGN, "gemm_nn: D not 16-byte aligned");
  Operand a{A, 0, M, K, K, 1, M * K};
  Operand b{B, 1, N, K, N, 1, N * K};   // stored (K, N): MN-major
  GemmParams p{};
  p.sched = SCHED_DENSE; p.b_mn = 1; p.M = (int)M; p.N = (int)N; p.K = (int)K; p.num_groups = 1;
  p.D = D; p.ldd = N; p.status = status;
  const int bn = pick_bn(N);
  Operand d{D, 0, M, N, N, 1, M * N};
  return dispatch_bn<EPI_STORE>(bn, a, b, &d, nullptr, p, (int)(ceil_div(M, BM) * ceil_div(N, bn)), (cudaStream_t)stream);
}

int b200moe_gemm_tn_splitk(const void* A, const void* B, float* P, int64_t M, int64_t N, int64_t K,
                           int64_t k_chunk, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(A && B && P, B200MOE_E_NULL, "gemm_tn_splitk: null pointer");
  CHECK_DIM8(M); CHECK_DIM8(N); CHECK_I32(M); CHECK_I32(N); CHECK_I32(K);
  B200_CHECK_ARG(k_chunk > 0 && k_chunk % 64 == 0, B200MOE_E_BAD_SHAPE,
                 "gemm_tn_splitk: k_chunk = %lld must be a positive multiple of 64", (long long)k_chunk);
  B200_CHECK_ARG(K > 0, B200MOE_E_BAD_SHAPE, "gemm_tn_splitk: K must be positive");
  B200_CHECK_ARG(aligned16(P), B200MOE_E_ALIGN, "gemm_tn_splitk: P not 16-byte aligned");
  const long long slices = ceil_div(K, k_chunk);
  Operand a{A, 1, M, K, M, 1, M * K};   // stored (K, M)
  Operand b{B, 1, N, K, N, 1, N * K};   // stored (K, N)
  GemmParams p{};
  p.sched = SCHED_GROUPED_K; p.a_mn = 1; p.b_mn = 1; p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.num_groups = (int)slices; p.k_chunk = (int)k_chunk; p.poffs = nullptr;
  p.D = P; p.ldd = N; p.d_group_stride = M * N; p.status = status;
  // Up to 128 rows the second half of a pair tile would multiply nothing but padding: single-CTA tiles.  us, 256-wide pair /
  // 128-wide tiles, 16 384 tokens: 16 x 2048 22.8 / 14.0, 64 x 2048 24.7 / 15.1, 128 x 512 19.1 / 8.7; 1024 tokens, 128 x
  // 1024 16.1 / 6.5.
  const int bn = M <= BM ? std::min(pick_bn(N), 128)
                         : pick_bn_grouped(N, 64, slices * ceil_div(M, 256), slices * ceil_div(M, BM));
  return dispatch_bn<EPI_STORE_F32>(bn, a, b, nullptr, nullptr, p, (int)(slices * ceil_div(M, BM) * ceil_div(N, bn)),
                                    (cudaStream_t)stream);
}

static int check_conv(const char* who, int64_t B, int64_t S, int64_t H, int64_t E, int taps, int64_t s_mult,
                      int64_t c_mult64) {
  B200_CHECK_ARG(B > 0 && S > 0 && taps >= 1 && taps <= 64, B200MOE_E_BAD_SHAPE, "%s: B = %lld, S = %lld, taps = %d", who,
                 (long long)B, (long long)S, taps);
  B200_CHECK_ARG(S % s_mult == 0, B200MOE_E_BAD_SHAPE, "%s: S = %lld must be a multiple of %lld", who, (long long)S,
                 (long long)s_mult);
  B200_CHECK_ARG(c_mult64 % 64 == 0, B200MOE_E_BAD_SHAPE, "%s: the convolved channel count %lld must be a multiple of 64",
                 who, (long long)c_mult64);
  B200_CHECK_ARG(H % 8 == 0 && E % 8 == 0 && H > 0 && E > 0, B200MOE_E_BAD_SHAPE, "%s: H = %lld, E = %lld", who,
                 (long long)H, (long long)E);
  B200_CHECK_ARG(B * S < (1LL << 31) && taps * H < (1LL << 31) && taps * E < (1LL << 31), B200MOE_E_BAD_SHAPE,
                 "%s: extent beyond 2^31", who);
  return 0;
}

int b200moe_conv_gemm_fwd(const void* x, const void* wf, void* logits, int64_t B, int64_t S, int64_t H, int64_t E, int taps,
                          int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(x && wf && logits, B200MOE_E_NULL, "conv_gemm_fwd: null pointer");
  int rc = check_conv("conv_gemm_fwd", B, S, H, E, taps, BM, H);
  if (rc) return rc;
  B200_CHECK_ARG(aligned16(logits), B200MOE_E_ALIGN, "conv_gemm_fwd: logits not 16-byte aligned");
  const int64_t M = B * S, K = taps * H;
  Operand a{x, 0, S, H, H, B, S * H};       // {H, S, B}: positions outside [0, S) read as zero
  Operand b{wf, 0, E, K, K, 1, E * K};
  GemmParams p{};
  p.sched = SCHED_DENSE; p.M = (int)M; p.N = (int)E; p.K = (int)K; p.num_groups = 1;
  p.D = logits; p.ldd = E; p.d_group_stride = S * E; p.status = status;
  p.conv_taps = taps; p.conv_S = (int)S; p.conv_C = (int)H; p.conv_sign = 1;
  const int bn = pick_bn(E);
  Operand d{logits, 0, S, E, E, B, S * E};
  return dispatch_bn<EPI_STORE, true>(bn, a, b, &d, nullptr, p, (int)(B * ceil_div(S, BM) * ceil_div(E, bn)), (cudaStream_t)stream);
}

int b200moe_conv_gemm_logits(const void* x, const void* weight_rows, void* logits, int64_t B, int64_t S, int64_t H, int64_t E,
                             int taps, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(x && weight_rows && logits, B200MOE_E_NULL, "conv_gemm_logits: null pointer");
  int rc = check_conv("conv_gemm_logits", B, S, H, E, taps, 1, 64);
  if (rc) return rc;
  B200_CHECK_ARG(H % 16 == 0, B200MOE_E_BAD_SHAPE, "conv_gemm_logits: H = %lld must be a multiple of 16", (long long)H);
  B200_CHECK_ARG(aligned16(logits), B200MOE_E_ALIGN, "conv_gemm_logits: logits not 16-byte aligned");
  Operand a{x, 0, S, H, H, B, S * H};                    // {H, S, B}: positions outside [0, S) read as zero
  Operand b{weight_rows, 0, E, H, H, taps, E * H};       // {H, E, taps}
  GemmParams p{};
  p.sched = SCHED_DENSE; p.M = (int)(B * S); p.N = (int)E; p.K = (int)(taps * ceil_div(H, BK) * BK); p.num_groups = 1;
  p.D = logits; p.ldd = E; p.d_group_stride = S * E; p.status = status;
  p.conv_taps = taps; p.conv_S = (int)S; p.conv_C = (int)H; p.conv_sign = 1; p.conv_b_taps = 1;
  const int bn = pick_bn(E);
  Operand d{logits, 0, S, E, E, B, S * E};
  return dispatch_bn<EPI_STORE, true>(bn, a, b, &d, nullptr, p, (int)(B * ceil_div(S, BM) * ceil_div(E, bn)), (cudaStream_t)stream);
}

int b200moe_conv_gemm_dx(const void* grad_logits, const void* wb, void* grad_x, int64_t B, int64_t S, int64_t H, int64_t E,
                         int taps, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(grad_logits && wb && grad_x, B200MOE_E_NULL, "conv_gemm_dx: null pointer");
  int rc = check_conv("conv_gemm_dx", B, S, H, E, taps, BM, E);
  if (rc) return rc;
  B200_CHECK_ARG(aligned16(grad_x), B200MOE_E_ALIGN, "conv_gemm_dx: grad_x not 16-byte aligned");
  const int64_t M = B * S, K = taps * E;
  Operand a{grad_logits, 0, S, E, E, B, S * E};   // {E, S, B}, read (taps - 1) - tap positions ahead
  Operand b{wb, 1, H, K, H, 1, H * K};            // stored (taps * E, H): MN-major
  GemmParams p{};
  p.sched = SCHED_DENSE; p.b_mn = 1; p.M = (int)M; p.N = (int)H; p.K = (int)K; p.num_groups = 1;
  p.D = grad_x; p.ldd = H; p.d_group_stride = S * H; p.status = status;
  p.conv_taps = taps; p.conv_S = (int)S; p.conv_C = (int)E; p.conv_sign = -1;
  const int bn = pick_bn(H);
  Operand d{grad_x, 0, S, H, H, B, S * H};
  return dispatch_bn<EPI_STORE, true>(bn, a, b, &d, nullptr, p, (int)(B * ceil_div(S, BM) * ceil_div(H, bn)), (cudaStream_t)stream);
}

int b200moe_conv_gemm_dw_splitk(const void* grad_logits, const void* x, float* P, int64_t B, int64_t S, int64_t H,
                                int64_t E, int taps, int64_t k_chunk, int32_t* status, b200moe_stream_t stream) {
  B200_CHECK_ARG(grad_logits && x && P, B200MOE_E_NULL, "conv_gemm_dw_splitk: null pointer");
  int rc = check_conv("conv_gemm_dw_splitk", B, S, H, E, taps, 64, H);
  if (rc) return rc;
  B200_CHECK_ARG(k_chunk > 0 && k_chunk % 64 == 0, B200MOE_E_BAD_SHAPE,
                 "conv_gemm_dw_splitk: k_chunk = %lld must be a positive multiple of 64", (long long)k_chunk);
  B200_CHECK_ARG(aligned16(P), B200MOE_E_ALIGN, "conv_gemm_dw_splitk: P not 16-byte aligned");
  const int64_t K = B * S, N = taps * H;
  const long long slices = ceil_div(K, k_chunk);
  Operand a{grad_logits, 1, E, K, E, 1, E * K};   // stored (B*S, E)
  Operand b{x, 1, H, S, H, B, S * H};             // {H, S, B}: the k rows of tap j are read j - (taps - 1) positions away
  GemmParams p{};
  p.sched = SCHED_GROUPED_K; p.a_mn = 1; p.b_mn = 1; p.M = (int)E; p.N = (int)N; p.K = (int)K;
  p.num_groups = (int)slices; p.k_chunk = (int)k_chunk; p.poffs = nullptr;
  p.D = P; p.ldd = N; p.d_group_stride = E * N; p.status = status;
  p.conv_taps = taps; p.conv_S = (int)S; p.conv_C = (int)H; p.conv_sign = 1;
  const int bn = H % 256 == 0 ? 256 : (H % 128 == 0 ? 128 : 64);   // a tile's columns belong to one tap
  return dispatch_bn<EPI_STORE_F32, true>(bn, a, b, nullptr, nullptr, p, (int)(slices * ceil_div(E, BM) * ceil_div(N, bn)),
                                    (cudaStream_t)stream);
}

int b200moe_expert_gate_up_swiglu(const void* x_s, const void* gate_up_proj, const int32_t* tile_expert,
                                  const int32_t* poffs, int64_t rows_cap, int E, int64_t H, int64_t I,
                                  void* gate_up, void* inter, int32_t* status, b200moe_stream_t stream) {
  return b200moe_expert_gate_up_act(x_s, gate_up_proj, nullptr, tile_expert, poffs, rows_cap, 0, 0, E, H, I, gate_up,
                                    inter, status, stream);
}

int b200moe_expert_gate_up_act(const void* x_s, const void* gate_up_proj, const int32_t* act_codes,
                               const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int64_t row_lo,
                               int64_t row_hi, int E, int64_t H, int64_t I, void* gate_up, void* inter,
                               int32_t* status, b200moe_stream_t stream) {
  return expert_gate_up(x_s, H, gate_up_proj, act_codes, tile_expert, poffs, rows_cap, row_lo, row_hi, E, H, I, gate_up, 2 * I, inter, I, status,
                        stream);
}

int b200moe_expert_linear(const void* a, const void* w, const int32_t* tile_expert, const int32_t* poffs,
                          int64_t rows_cap, int E, int64_t N, int64_t K, void* out, int32_t* status,
                          b200moe_stream_t stream) {
  return expert_linear(a, K, w, tile_expert, poffs, rows_cap, E, N, K, out, N, status, stream);
}

int b200moe_expert_gram(const void* x, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E,
                        int64_t K, int mirror, void* out, int32_t* status, b200moe_stream_t stream) {
  return expert_gram(x, tile_expert, poffs, rows_cap, E, K, mirror, E >= 1 ? rows_cap / E : 0, out, status, stream);
}

int b200moe_expert_linear_axpby(const void* a, const void* w, const void* c, float alpha, float beta, float diag,
                                int symmetric, const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E,
                                int64_t N, int64_t K, void* out, int32_t* status, b200moe_stream_t stream) {
  return expert_linear_axpby(a, w, c, alpha, beta, diag, symmetric, tile_expert, poffs, rows_cap, E, N, K, N, K, out, status, stream);
}

int b200moe_expert_linear_t(const void* a, const void* w, const int32_t* tile_expert, const int32_t* poffs,
                            int64_t rows_cap, int E, int64_t K, int64_t N, void* out, int32_t* status,
                            b200moe_stream_t stream) {
  return expert_linear_t(a, K, w, tile_expert, poffs, rows_cap, E, K, N, K, out, N, status, stream);
}

int b200moe_expert_linear_push(const void* a, const void* w, int w_kn, const int32_t* tile_expert, const int32_t* poffs,
                               int64_t rows_cap, int E, int64_t N, int64_t K, const int32_t* row_rank,
                               const int32_t* row_slot, const int64_t* peer_base, int32_t* status,
                               b200moe_stream_t stream) {
  int rc = check_grouped("expert_linear_push", a, w, peer_base, tile_expert, poffs, rows_cap, E, N, K);
  if (rc) return rc;
  B200_CHECK_ARG(tile_expert && row_rank && row_slot && peer_base, B200MOE_E_NULL, "expert_linear_push: null pointer");
  B200_CHECK_ARG(N % 64 == 0, B200MOE_E_BAD_SHAPE, "expert_linear_push: N = %lld must be a multiple of 64", (long long)N);
  Operand oa{a, 0, rows_cap, K, K, 1, rows_cap * K};
  Operand ob_nk{w, 0, N, K, K, E, N * K};   // W (E, N, K): rows = output columns
  Operand ob_kn{w, 1, N, K, N, E, K * N};   // W[e] stored (K, N): MN-major
  GemmParams p{};
  p.sched = SCHED_GROUPED_M; p.b_mn = w_kn ? 1 : 0; p.N = (int)N; p.K = (int)K; p.num_groups = E;
  p.tile_expert = tile_expert; p.poffs = poffs; p.D = nullptr; p.ldd = N; p.status = status;
  p.push_rank = row_rank; p.push_slot = row_slot; p.push_base = reinterpret_cast<const long long*>(peer_base);
  return dispatch_bn<EPI_STORE>(256, oa, w_kn ? ob_kn : ob_nk, nullptr, nullptr, p, 0, (cudaStream_t)stream);
}

int b200moe_expert_down(const void* inter, const void* down_proj, const int32_t* tile_expert, const int32_t* poffs,
                        int64_t rows_cap, int E, int64_t H, int64_t I, void* eo, int32_t* status,
                        b200moe_stream_t stream) {
  return b200moe_expert_linear(inter, down_proj, tile_expert, poffs, rows_cap, E, H, I, eo, status, stream);
}

int b200moe_expert_down_dgrad_glu(const void* grad_eo, const void* down_proj, const void* gate_up,
                                  const int32_t* tile_expert, const int32_t* poffs, int64_t rows_cap, int E,
                                  int64_t H, int64_t I, void* grad_gate_up, int32_t* status,
                                  b200moe_stream_t stream) {
  return b200moe_expert_down_dgrad_act(grad_eo, down_proj, gate_up, nullptr, tile_expert, poffs, rows_cap, 0, 0, E, H, I,
                                       grad_gate_up, status, stream);
}

int b200moe_expert_down_dgrad_act(const void* grad_eo, const void* down_proj, const void* gate_up,
                                  const int32_t* act_codes, const int32_t* tile_expert, const int32_t* poffs,
                                  int64_t rows_cap, int64_t row_lo, int64_t row_hi, int E, int64_t H, int64_t I,
                                  void* grad_gate_up, int32_t* status, b200moe_stream_t stream) {
  return expert_down_dgrad(grad_eo, H, down_proj, gate_up, 2 * I, act_codes, tile_expert, poffs, rows_cap, row_lo, row_hi, E, H, I, grad_gate_up,
                           status, stream);
}

int b200moe_expert_gate_up_dgrad(const void* grad_gate_up, const void* gate_up_proj, const int32_t* tile_expert,
                                 const int32_t* poffs, int64_t rows_cap, int E, int64_t H, int64_t I,
                                 void* grad_x_s, int32_t* status, b200moe_stream_t stream) {
  return b200moe_expert_linear_t(grad_gate_up, gate_up_proj, tile_expert, poffs, rows_cap, E, 2 * I, H, grad_x_s,
                                 status, stream);
}

int b200moe_expert_wgrad(const void* A, const void* B, const int32_t* poffs, const int32_t* counts, int64_t rows_cap,
                         int E, int64_t Na, int64_t Nb, void* out, int32_t* status, b200moe_stream_t stream) {
  return expert_wgrad(A, Na, B, Nb, poffs, counts, rows_cap, E, Na, Nb, out, status, stream);
}

}  // extern "C"
