// Grouped GEMM: several independent products with a common reduction length in ONE persistent launch.
//
//   D_p [M_p, N_p] (fp32) (+)= alpha * A_p . B_p      p = 0 .. n-1,  same K, same operand layouts
//
// Purpose: the four weight gradients of a transformer block (dW = dY^T X with K = tokens) have 12 - 48
// output tiles each, far fewer than the 74 CTA pairs, so on their own they need split-K plus a reduction kernel.
// Together they are 72 tiles of 256 x 384 or 144 of 256 x 192: one or two full waves with no split at all - every output element
// is reduced over K by one CTA pair in k-block order, which is also the simplest deterministic order there is.
//
// The kernel is the CTA-pair tcgen05 GEMM of gemm2_kernel.cuh with a table of problems in the place of one: a work
// item is (problem, n tile, m tile), items are dealt round robin to the pairs, and each problem brings its own pair of
// tensor maps.  Its outputs are fp32 with optional accumulation; no bias, activation, residual, split or collective.
// The reference has no grouped product (its CPU `mod gemm`, ft-kernel-cpu/src/lib.rs:18-1677, runs one
// matrix product per call).
#pragma once
#include "gemm2_kernel.cuh"

namespace ftk {

constexpr int GG_MAX = 8;   // problems per launch
constexpr int GG_BN = 192, GG_BN_WIDE = 384;

struct GroupArgs {
  int n;                       // number of problems
  int K;
  int a_mn, b_mn;
  int M[GG_MAX], N[GG_MAX];
  int tile_end[GG_MAX];        // running total of tiles up to and including problem p
  float* D[GG_MAX];
  long long ldd[GG_MAX];
  int accumulate[GG_MAX];
  FastDiv by_tiles_m[GG_MAX];
  float alpha;
  int* status;
};
struct GroupMaps {
  CUtensorMap a[GG_MAX];
  CUtensorMap b[GG_MAX];
};

struct GroupTile {
  int p, m_t, n_t;
};
__device__ __forceinline__ GroupTile group_decode(int item, const GroupArgs& g) {
  GroupTile t;
  t.p = 0;
#pragma unroll
  for (int i = 0; i < GG_MAX - 1; ++i)
    if (i + 1 < g.n && item >= g.tile_end[i]) t.p = i + 1;
  const int local = item - (t.p > 0 ? g.tile_end[t.p - 1] : 0);
  t.n_t = g.by_tiles_m[t.p].div(local);
  t.m_t = local - t.n_t * (int)g.by_tiles_m[t.p].d;
  return t;
}

// KIND: EPI_KIND_F32, or EPI_KIND_ANY when an output's rows are not made of aligned 16-byte segments.
// BN = 192: two accumulators, the epilogue of a tile under the main loop of the next.  BN = 384: one accumulator.
template <int BN, int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G_THREADS, 1)
gemm_group_bf16_sm100_kernel(const __grid_constant__ GroupMaps maps, const GroupArgs g) {
  using Cfg = PairCfg<BN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(g.status, 0, FT_ERR_BAD_ARG);
    return;
  }
  PairCta<BN> cta(smem);
  const int warp = cta.warp, lane = cta.lane, rank = cta.rank;
  WaitCtx ctx{g.status, cta.abort_f};
  cta.setup();
  pdl_wait();
  if (warp != 0) pdl_trigger();      // (these warps have seen the tensor-memory allocation)

  const int pair = (int)blockIdx.x >> 1;
  const int n_pairs = (int)gridDim.x >> 1;
  const int total = g.tile_end[g.n - 1];
  const int kblocks = (g.K + G_BK - 1) / G_BK;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int item = pair; ok && item < total; item += n_pairs) {
      const GroupTile t = group_decode(item, g);
      const CUtensorMap* mapA = &maps.a[t.p];
      const CUtensorMap* mapB = &maps.b[t.p];
      if (lane == 0) {
        tma_prefetch_desc(mapA);
        tma_prefetch_desc(mapB);
      }
      const int a_row = (2 * t.m_t + rank) * G_BM, b_row = t.n_t * BN + rank * Cfg::HALF;
      for (int kb = 0; kb < kblocks; ++kb) {
        if (!mbar_wait_warp(&cta.empty[s], ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) {
          ok = false;
          break;
        }
        if (elect_one()) cta.load(s, mapA, mapB, g.a_mn, g.b_mn, kb, a_row, b_row, 0, 0);
        __syncwarp();
        if (++s == Cfg::STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0) {
      int s = 0;
      uint32_t ph = 0;
      int acc = 0;
      uint32_t acc_ph = 0;
      for (int item = pair; item < total; item += n_pairs) {
        if (!mbar_wait_warp(&cta.tempty[acc], ((acc_ph >> acc) & 1u) ^ 1u, ctx, FT_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        if (!cta.mma_tile(cta.tmem_base + acc * Cfg::ACC_STRIDE, 0, kblocks, g.a_mn, g.b_mn, &cta.tfull[acc], s, ph, ctx))
          break;
        acc_ph ^= (1u << acc);
        if (Cfg::ACCS > 1) acc ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (8 warps, both CTAs): fp32 store / accumulate
    const int ew = warp - 2;
    const int q = warp & 3;
    const int half = ew >> 2;             // column half of the tile
    GemmArgs p;
    p.L0 = p.L1 = p.splits = p.out_fp32 = 1;
    p.d_s0 = p.d_s1 = p.ldr = p.r_s0 = p.r_s1 = 0;
    p.bias = p.resid = nullptr;
    p.aux = nullptr;
    p.ws = nullptr;
    p.alpha = g.alpha;
    p.epi = FTK_EPI_NONE;
    TileEpilogue<KIND> epi(p, smem + Cfg::OFF_STAGE + ew * EPI_STAGE_BYTES,
                     reinterpret_cast<__nv_bfloat16*>(smem + Cfg::OFF_BIAS + ew * EPI_BIAS_BYTES), lane);
    int acc = 0;
    uint32_t acc_ph = 0;
    for (int item = pair; item < total; item += n_pairs) {
      const GroupTile t = group_decode(item, g);
      p.M = g.M[t.p];
      p.N = g.N[t.p];
      p.D = g.D[t.p];
      p.ldd = g.ldd[t.p];
      p.accumulate = g.accumulate[t.p];
      const int row = (2 * t.m_t + rank) * G_BM + q * 32, col = t.n_t * BN + half * (BN / 2);
      constexpr int FIRST = BN > 256 ? 4 : Cfg::C_HALF;      // chunks of this warp beside one another in tensor memory
      epi.begin(0, 0, row, col, FIRST, false);
      if (!mbar_wait(&cta.tfull[acc], (acc_ph >> acc) & 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&cta.tempty[acc]);
      };
      const uint32_t lanes = cta.tmem_base + ((uint32_t)(q * 32) << 16);
      if constexpr (BN > 256) {
        // the tile's halves are [0, 128) and [256, 320) of the accumulator, [128, 256) and [320, 384)
        epi.run(lanes + half * 128, FIRST, [] {});
        epi.begin(0, 0, row, col + 128, Cfg::C_HALF - FIRST, false);
        epi.run(lanes + 256 + half * ((BN - 256) / 2), Cfg::C_HALF - FIRST, release);
      } else {
        epi.run(lanes + acc * Cfg::ACC_STRIDE + half * (BN / 2), FIRST, release);
      }
      acc_ph ^= (1u << acc);
      if (Cfg::ACCS > 1) acc ^= 1;
    }
  }
  cta.teardown();
}

}  // namespace ftk
