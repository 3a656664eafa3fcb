// bf16 GEMM on CTA pairs (tcgen05 cta_group::2): one 256 x BN output tile per 2-CTA cluster, BN = 128 to 256 in steps of 32.
//
// Each CTA of the pair loads its own 128 rows of A and its own BN / 2 columns of B per k-block
// (32 KB per stage at BN = 256 instead of the 48 KB a lone 128 x 256 tile needs), which cuts the L2 -> SM
// operand traffic per FLOP by a third - the limiter of the single-CTA kernel.  The leader CTA
// (cluster rank 0) issues MMAs that read both CTAs' shared memory and write 128 accumulator rows
// x BN columns into each CTA's TMEM; both CTAs run a TMA producer warp and 8 epilogue warps.
// TMA completion bytes of both CTAs go to the leader's `full` barrier; `empty` / `tmem full` are
// signalled in both CTAs by a commit multicast (no data multicast anywhere); the peer's
// epilogue releases accumulators with remote arrives on the leader's `tmem empty` barrier.
//
// The narrower tiles exist for the tail: 74 pairs walk whole tiles, and 8192 x 768 is 96 tiles of 256 x 256 (1.3 waves,
// so 2) but 128 of 256 x 192 (1.7 waves of 3/4 of the work); 1500 x 1280 is 30 tiles of 256 x 256 but 60 of 256 x 128.
//
// Same operand forms (K-major / MN-major), epilogues and deterministic split-K as the single-CTA
// kernel in gemm_kernel.cuh; the k order of every output element is ascending and independent
// of the grid and of the tile width.
#pragma once
#include "gemm_kernel.cuh"

namespace ftk {

// The parts of a pair kernel that do not depend on where its tiles come from: shared-memory layout, barriers, one
// k-block of loads, one k-block of MMAs.
template <int BN_>
struct PairCfg {
  static constexpr int BN = BN_;                   // tile columns (BN / 2 staged per CTA)
  static constexpr int HALF = BN / 2;
  static constexpr int MN_CHUNKS = (HALF + 63) / 64;   // 64-column boxes of an MN-major B half (a half of 80, 96 or 112 loads 128 columns)
  static constexpr int A_BYTES = G_BM * G_BK * 2;  // per CTA and stage
  static constexpr int B_BYTES = MN_CHUNKS * 64 * G_BK * 2;
  static constexpr int STAGES = BN == 384 ? 4 : (BN == 128 ? 8 : 6);
  static constexpr int ACCS = BN > 256 ? 1 : 2;    // accumulators
  static constexpr int ACC_STRIDE = BN == 128 ? 128 : 256;
  static constexpr int TMEM_COLS = BN == 128 ? 256 : 512;
  static constexpr int OFF_BARS = STAGES * (A_BYTES + B_BYTES);
  static constexpr int OFF_STAGE = OFF_BARS + 256;
  static constexpr int OFF_BIAS = OFF_STAGE + G_EPI_WARPS * EPI_STAGE_BYTES;
  static constexpr int SMEM = OFF_BIAS + G_EPI_WARPS * EPI_BIAS_BYTES;
  static constexpr int CHUNKS = BN / 32;
  static constexpr int C_HALF = (CHUNKS + 1) / 2;    // chunks of the first four epilogue warps, the others take the rest
  static_assert((2 * STAGES + 4) * 8 + 8 <= 256, "barrier space");
  static_assert(SMEM <= 232448, "shared memory");
};

template <int BN>
struct PairCta {
  using Cfg = PairCfg<BN>;
  uint8_t *sA, *sB, *smem;
  uint64_t *full, *empty, *tfull, *tempty;     // `full` and `tempty`: the leader's copies are the ones in use
  uint32_t* tmem_slot;
  int* abort_f;
  int warp, lane, rank;
  uint32_t tmem_base;

  __device__ __forceinline__ explicit PairCta(uint8_t* s) : smem(s) {
    sA = smem;
    sB = smem + Cfg::STAGES * Cfg::A_BYTES;
    full = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BARS);
    empty = full + Cfg::STAGES;
    tfull = empty + Cfg::STAGES;
    tempty = tfull + 2;
    tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    abort_f = reinterpret_cast<int*>(tmem_slot + 1);
    warp = warp_index();
    lane = threadIdx.x & 31;
    rank = (int)cluster_ctarank();
  }
  // The producer warp leaves as soon as both CTAs' barriers exist; tensor memory is allocated behind its first loads.
  __device__ __forceinline__ void setup() {
    if (threadIdx.x == 0) {
      for (int i = 0; i < Cfg::STAGES; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tfull[i], 1);
        mbar_init(&tempty[i], 2 * G_EPI_WARPS);
      }
      *abort_f = 0;
      fence_mbar_init();
    }
    __syncwarp();
    cluster_arrive();
    if (warp == 1) {
      tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish_pair();
    }
    cluster_wait();
    if (warp != 0) {
      tc_fence_before();
      setup_barrier(G_THREADS - 32);
      tc_fence_after();
      tmem_base = *tmem_slot;
    }
  }
  // k-block `kb` of the tile at (a_row, b_row): this CTA's half of both operands into stage s (one lane).
  __device__ __forceinline__ void load(int s, const CUtensorMap* tmA, const CUtensorMap* tmB, int a_mn, int b_mn, int kb,
                                       int a_row, int b_row, int l0, int l1) {
    // the leader's barrier collects the bytes of both CTAs
    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * (Cfg::A_BYTES + (b_mn ? Cfg::B_BYTES : Cfg::HALF * G_BK * 2)));
    uint8_t* a_dst = sA + s * Cfg::A_BYTES;
    uint8_t* b_dst = sB + s * Cfg::B_BYTES;
    if (!a_mn) {
      tma_load_4d_pair(a_dst, tmA, &full[s], kb * G_BK, a_row, l0, l1);
    } else {
#pragma unroll
      for (int cc = 0; cc < G_BM / 64; ++cc)
        tma_load_4d_pair(a_dst + cc * (G_BK * 128), tmA, &full[s], a_row + cc * 64, kb * G_BK, l0, l1);
    }
    if (!b_mn) {
      tma_load_4d_pair(b_dst, tmB, &full[s], kb * G_BK, b_row, l0, l1);
    } else {
#pragma unroll
      for (int cc = 0; cc < Cfg::MN_CHUNKS; ++cc)
        tma_load_4d_pair(b_dst + cc * (G_BK * 128), tmB, &full[s], b_row + cc * 64, kb * G_BK, l0, l1);
    }
  }
  // The MMA loop of one tile over k-blocks [kb0, kb1): leader CTA, whole warp.  Returns false on an abort.
  __device__ __forceinline__ bool mma_tile(uint32_t d_tmem, int kb0, int kb1, int a_mn, int b_mn, uint64_t* done, int& s,
                                           uint32_t& ph, const WaitCtx& ctx) {
    // (an instruction has 256 columns at most: a wider tile takes the first 128 columns of both halves, then the rest)
    const uint32_t idesc = make_idesc_bf16(2 * G_BM, BN > 256 ? 256 : BN, a_mn, b_mn);
    const uint32_t idesc2 = make_idesc_bf16(2 * G_BM, BN > 256 ? BN - 256 : 64, a_mn, b_mn);
    const uint32_t a_lbo = a_mn ? G_BK * 128 : 16, a_adv16 = (a_mn ? G_UMMA_K * 128 : G_UMMA_K * 2) >> 4;
    const uint32_t b_lbo = b_mn ? G_BK * 128 : 16, b_adv16 = (b_mn ? G_UMMA_K * 128 : G_UMMA_K * 2) >> 4;
    const uint32_t a_lo0 = desc_lo(smem_u32(sA), a_lbo), b_lo0 = desc_lo(smem_u32(sB), b_lbo);
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full[s], ph, ctx, FT_ERR_WAIT_FULL)) return false;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_lo = a_lo0 + (uint32_t)s * (Cfg::A_BYTES >> 4);
        const uint32_t b_lo = b_lo0 + (uint32_t)s * (Cfg::B_BYTES >> 4);
        umma_bf16_pair_lo(d_tmem, a_lo, b_lo, idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
        for (int k = 1; k < G_BK / G_UMMA_K; ++k)
          umma_bf16_pair_lo(d_tmem, a_lo + k * a_adv16, b_lo + k * b_adv16, idesc, 1u);
        if constexpr (BN > 256) {
          const uint32_t b2_lo = b_lo + (128 * G_BK * 2 >> 4);      // K-major: row 128; MN-major: the third 64-column box
          umma_bf16_pair_lo(d_tmem + 256, a_lo, b2_lo, idesc2, kb > kb0 ? 1u : 0u);
#pragma unroll
          for (int k = 1; k < G_BK / G_UMMA_K; ++k)
            umma_bf16_pair_lo(d_tmem + 256, a_lo + k * a_adv16, b2_lo + k * b_adv16, idesc2, 1u);
        }
        umma_commit_pair(&empty[s], 3);                       // the stage is free in both CTAs
        if (kb == kb1 - 1) umma_commit_pair(done, 3);         // both epilogues may drain
      }
      __syncwarp();
      if (++s == Cfg::STAGES) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (kb1 <= kb0 && elect_one()) umma_commit_pair(done, 3);   // empty split
    __syncwarp();
    return true;
  }
  __device__ __forceinline__ void teardown() {
    if (*abort_f) {
      for (int i = 0; i < 100; ++i) __nanosleep(10000);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither CTA leaves while the other may still signal it
    if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  }
};

// Tile t of a product: groups of by_gm.d m tiles, within a group m fastest, then n (the host's set_pair_groups has the reason).
__device__ __forceinline__ void pair_tile(const GemmArgs& p, int t, int tiles_m2, int& m_t, int& n_t) {
  const int g = p.by_group.div(t), r = t - g * (int)p.by_group.d, m0 = g * (int)p.by_gm.d;
  const bool full = m0 + (int)p.by_gm.d <= tiles_m2;
  n_t = full ? p.by_gm.div(r) : p.by_gm_last.div(r);
  m_t = m0 + r - n_t * (int)(full ? p.by_gm.d : p.by_gm_last.d);
}

template <int BN, int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G_THREADS, 1)
gemm2_bf16_sm100_kernel(const __grid_constant__ CUtensorMap tmA,
                        const __grid_constant__ CUtensorMap tmB, const GemmArgs p) {
  using Cfg = PairCfg<BN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  // (the dynamic shared-memory base has the same offset in both CTAs, so both take the same branch)
  if ((smem_u32(smem) & 1023u) != 0u) {
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(p.status, 0, FT_ERR_BAD_ARG);
    return;
  }
  PairCta<BN> cta(smem);
  const int warp = cta.warp, lane = cta.lane, rank = cta.rank;
  WaitCtx ctx{p.status, cta.abort_f};
  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  cta.setup();
  pdl_wait();
  if (warp != 0) pdl_trigger();      // (these warps have seen the tensor-memory allocation)

  const int pair = (int)blockIdx.x >> 1;
  const int n_pairs = (int)gridDim.x >> 1;
  const int tiles_m2 = (int)p.by_tiles_m.d, tiles_mn = (int)p.by_tiles_mn.d, nbatch = (int)p.by_batches.d;
  const int total = tiles_mn * nbatch * p.splits;
  const int kblocks_all = (p.K + G_BK - 1) / G_BK;
  const int kb_per_split = p.splits > 1 ? (kblocks_all + p.splits - 1) / p.splits : kblocks_all;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int item = pair; ok && item < total; item += n_pairs) {
      const int sl = p.by_tiles_mn.div(item), t = item - sl * tiles_mn;      // (split, batch), tile
      const int sp = p.by_batches.div(sl), l = sl - sp * nbatch;
      int m_t, n_t;
      pair_tile(p, t, tiles_m2, m_t, n_t);
      const int a_row = (2 * m_t + rank) * G_BM;
      const int b_row = n_t * BN + rank * Cfg::HALF;
      const int l1 = p.by_l0.div(l), l0 = l - l1 * p.L0;
      const int kb0 = sp * kb_per_split;
      const int kb1 = min(kblocks_all, kb0 + kb_per_split);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(&cta.empty[s], ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) {
          ok = false;
          break;
        }
        if (elect_one()) cta.load(s, &tmA, &tmB, p.a_mn, p.b_mn, kb, a_row, b_row, l0, l1);
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
        const int kb0 = p.by_batches.div(p.by_tiles_mn.div(item)) * kb_per_split;
        const int kb1 = min(kblocks_all, kb0 + kb_per_split);
        if (!mbar_wait_warp(&cta.tempty[acc], ((acc_ph >> acc) & 1u) ^ 1u, ctx, FT_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        if (!cta.mma_tile(cta.tmem_base + acc * Cfg::ACC_STRIDE, kb0, kb1, p.a_mn, p.b_mn, &cta.tfull[acc], s, ph, ctx))
          break;
        acc_ph ^= (1u << acc);
        acc ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (8 warps, both CTAs)
    const int ew = warp - 2;
    const int q = warp & 3;
    const int c_begin = (ew >> 2) * Cfg::C_HALF, chunks = (ew >> 2) ? Cfg::CHUNKS - Cfg::C_HALF : Cfg::C_HALF;
    TileEpilogue<KIND> epi(p, smem + Cfg::OFF_STAGE + ew * EPI_STAGE_BYTES,
                     reinterpret_cast<__nv_bfloat16*>(smem + Cfg::OFF_BIAS + ew * EPI_BIAS_BYTES), lane);
    int acc = 0;
    uint32_t acc_ph = 0;
    for (int item = pair; item < total; item += n_pairs) {
      const int sl = p.by_tiles_mn.div(item), t = item - sl * tiles_mn;
      const int sp = p.by_batches.div(sl), l = sl - sp * nbatch;
      int m_t, n_t;
      pair_tile(p, t, tiles_m2, m_t, n_t);
      epi.begin(sp, l, (2 * m_t + rank) * G_BM + q * 32, n_t * BN + c_begin * 32, chunks,
                sp * kb_per_split >= kblocks_all);
      if (!mbar_wait(&cta.tfull[acc], (acc_ph >> acc) & 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      epi.run(cta.tmem_base + acc * Cfg::ACC_STRIDE + c_begin * 32 + ((uint32_t)(q * 32) << 16), chunks, [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&cta.tempty[acc]);   // the MMA warp lives in the leader CTA
      });
      acc_ph ^= (1u << acc);
      acc ^= 1;
    }
  }
  cta.teardown();
}

}  // namespace ftk
