// Flash attention backward for sm_100a on tcgen05/TMEM, head_dim 64/128.
//
// Semantics (reference: ft-kernel-cpu/src/lib.rs:5300 sdpa_backward_f64; forward in
// ft-kernel-cpu/src/lib.rs:4572): P is recomputed from the saved log-sum-exp, then
//   dV = P^T dO, dP = dO V^T, dS = P o (dP - rowsum(dO o O)), dQ = scale dS K,
//   dK = scale dS^T Q.
//
// Layout: Q/K/V/O/dO are addressed in place inside the packed [B*S, 3*d] / [B*S, d]
// activations through 4-D TMA maps {head_dim, S, H, B}; no head split/merge copies.
//
// Two kernels, each 19 warps: warps 0-15 do the elementwise math, warp 16 is the TMA
// producer, warp 17 issues the score products (and owns TMEM), warp 18 the accumulating
// products - but for dK / dV with head_dim 128, where the four products of a block follow one another and warp 17 issues
// them all.  The 16 math warps split every 128 x 128 score tile by columns (four groups of 32
// columns; a thread owns one tile row inside its group's columns), so one tcgen05.ld per
// operand brings a thread's whole share into registers, the TMEM score tiles are released at
// once and the tensor core computes the next block's scores under the exponentials of this
// one.  P^T and dS go back to the tensor core through tensor memory (tcgen05.st by the row's thread, MMA with its A operand in
// TMEM), dS^T too with head_dim 64; with head_dim 128 the accumulators leave no columns for dS^T, which goes through
// 128B-swizzled bf16 tiles in shared memory.
//
// Determinism: dQ is accumulated in TMEM by the CTA that owns the query block (first kernel, which also writes
// delta = rowsum(dO o O)), dK / dV by the CTA that owns the key block, all in ascending block order; there are no atomics, so
// gradients are bit-identical run to run.
#include "attn_common.cuh"

namespace ftk {

constexpr int BW_THREADS = 608;
constexpr int BW_MATH = 16;         // one arrival per math warp on the math barriers
constexpr int BW_WARP_TMA = 16;
constexpr int BW_WARP_MMA = 17;      // issues the score products, owns TMEM
constexpr int BW_WARP_MMA2 = 18;     // issues the accumulating products (idle in dK / dV with head_dim 128)

// Store 32 packed-bf16 columns (16 words) of one tile row into the swizzled K-major tile.
__device__ __forceinline__ void store_row32_packed(uint8_t* tile, int row, int col0,
                                                   const uint32_t* w) {
  uint8_t* base = tile + (col0 >> 6) * AT_REGION + row * 128;
  const int j0 = (col0 & 63) >> 3;
#pragma unroll
  for (int t = 0; t < 4; ++t)
    *reinterpret_cast<uint4*>(base + (((j0 + t) ^ (row & 7)) << 4)) =
        make_uint4(w[4 * t], w[4 * t + 1], w[4 * t + 2], w[4 * t + 3]);
}
// One warp's 32 rows x 32 columns of an output: scaled fp32 accumulator rows (a thread owns one) as bf16 into the 2 KB `box`,
// laid out as the TMA's 64-byte swizzle has it, and from there to (col, row0) by the TMA unit, which cuts off the rows past the end.
// The box is free again behind bulk_wait_read_all() of lane 0.  (Four lanes writing 64 bytes of a row took 16 warps ~2000
// cycles; straight from its thread, a row 12 KB from the next costs 32 line accesses per instruction.)
__device__ __forceinline__ void store_out32(uint8_t* box, int lane, const uint32_t* r, float scale, const CUtensorMap* tm, int col,
                                            int row0, int h, int b, int S) {
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = pack_bf16(__uint_as_float(r[8 * t + 2 * i]) * scale, __uint_as_float(r[8 * t + 2 * i + 1]) * scale);
    *reinterpret_cast<uint4*>(box + lane * 64 + ((t ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0 && row0 < S) tma_store_4d(tm, box, col, row0, h, b);
}
constexpr int BW_BOX = 2048;
struct DkvMaps {
  CUtensorMap m[2];      // dV, dK
};

// =============================================================================== backward: dK, dV
template <int HD>
struct DkvCfg {
  static constexpr int TILE = (HD / 64) * AT_REGION;
  // head_dim 64 leaves 128 TMEM columns free: P^T and dS^T (packed bf16, 64 columns each) are
  // written there by the threads that own their rows, and the dV / dK products read their A
  // operand from tensor memory, so neither tile crosses shared memory (which a 128-row CTA tile
  // already saturates with its B operands).  head_dim 128 fills all 512 columns with
  // accumulators: P^T takes the place of the scores it was made from, dS^T is staged in shared
  // memory, and the two Q / dO stages that this leaves room for keep a load ahead of every block (with one stage and both
  // tiles in shared memory a block took ~6000 cycles, 2500 of them waiting for that load).
  static constexpr bool TS = (HD == 64);
  static constexpr int STAGES = (HD == 64) ? 3 : 2;          // Q / dO ring
  static constexpr int KVB = (HD == 64) ? 2 : 1;             // K / V buffers (one per work item)
  static constexpr int OFF_KV = 0;                           // [KVB] K, V
  static constexpr int OFF_Q = KVB * 2 * TILE;               // [STAGES]
  static constexpr int OFF_DO = OFF_Q + STAGES * TILE;       // [STAGES]
  static constexpr int OFF_DST = OFF_DO + STAGES * TILE;     // dS^T [keys x queries] (not TS), output staging
  static constexpr int OFF_STAT = OFF_DST + 2 * AT_REGION;   // [STAGES][2][128] floats
  static constexpr int OFF_BAR = OFF_STAT + STAGES * 2 * 128 * 4;
  static constexpr int SMEM = OFF_BAR + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_ST = 0, TM_DPT = 128, TM_DV = 256, TM_DK = 256 + HD;
  static constexpr int TM_PT = TS ? 256 + 2 * HD : TM_ST, TM_DST = 256 + 2 * HD + 64;   // TM_DST: TS only
  static_assert(SMEM <= 232448, "shared memory");
};

// One persistent CTA per SM walks (key block, head, batch) items; every ring and every barrier runs on across items, so the
// loads and the first score products of an item are issued under the last block and the output of the one before.  With one
// CTA per item, set-up, first loads and output were ~15000 cycles per item against 1800 per block.
template <int HD, bool LATE>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const __grid_constant__ DkvMaps out, const AttnArgs p) {
  using C = DkvCfg<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* kv_full = bars;         // [2]
  uint64_t* kv_empty = bars + 2;    // [2] the item's score products are done
  uint64_t* q_full = bars + 4;      // [4] Q tile and the block's statistics
  uint64_t* q_empty = bars + 8;     // [4]
  uint64_t* do_full = bars + 12;    // [4]
  uint64_t* do_empty = bars + 16;   // [4] head_dim 128: dO is done with after dV, half a block before Q
  uint64_t* st_full = bars + 20;    // S^T and dP^T in TMEM
  uint64_t* st_free = bars + 21;    // both copied to registers (one arrival per warp)
  uint64_t* pt_ready = bars + 22;   // P^T handed to the tensor core (one arrival per warp); TS: P^T and dS^T
  uint64_t* ds_ready = bars + 23;   // dS^T in shared memory (not TS)
  uint64_t* dv_done = bars + 24;    // dV product of the block done (not TS)
  uint64_t* acc_done = bars + 25;   // dV and dK products of the block done
  uint64_t* acc_free = bars + 26;   // the item's dV / dK copied to registers (one arrival per warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  int* abort_f = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  WaitCtx ctx{p.status, abort_f};

  if ((smem_u32(smem) & 1023u) != 0u) {
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(p.status, 0, FT_ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    mbar_init(st_full, 1);
    mbar_init(st_free, BW_MATH);
    mbar_init(pt_ready, BW_MATH);
    mbar_init(ds_ready, BW_MATH);
    mbar_init(dv_done, 1);
    mbar_init(acc_done, 1);
    mbar_init(acc_free, BW_MATH);
    *abort_f = 0;
    fence_mbar_init();
  }
  if (warp == BW_WARP_TMA && elect_one()) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == BW_WARP_MMA) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  const int n_hb = p.H * p.B;
  const int nq_all = (p.S + AT_T - 1) / AT_T;
  float* stat = reinterpret_cast<float*>(smem + C::OFF_STAT);
  TileWalk walk(p.n_tiles);

  if (warp == BW_WARP_TMA) {
    Ring<C::STAGES> rq;
    Ring<C::KVB> rk;
    bool ok = true;
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const int kb = p.by_hb.div(item), hb = item - kb * n_hb, b = p.by_h.div(hb), h = hb - b * p.H;
      const int qb_first = p.causal ? kb : 0, nit = nq_all - qb_first;
      // Per-query statistics (-lse and -delta) of a block travel with its Q / dO tiles: they are
      // fetched into registers one iteration ahead, so their global-memory latency is spent while
      // this warp waits for the stage, not between the stage becoming free and its TMA loads.
      const long long sbase = ((long long)b * p.H + h) * p.S;
      // (signs are changed where the values are stored: an operation on a value in flight would wait for it here)
      float lse_r[4], dl_r[4];
      auto fetch_stats = [&](int it) {
        const int q0 = (qb_first + it) * AT_T;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int gq = q0 + lane + 32 * u;
          lse_r[u] = INFINITY;
          dl_r[u] = 0.f;
          if (gq < p.S) {
            lse_r[u] = p.lse[sbase + gq];
            dl_r[u] = p.delta[sbase + gq];
          }
        }
      };
      fetch_stats(0);
      if (!mbar_wait_warp(&kv_empty[rk.s], rk.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) break;
      if (elect_one()) {
        uint8_t* kv = smem + C::OFF_KV + rk.s * 2 * C::TILE;
        mbar_arrive_expect_tx(&kv_full[rk.s], 2 * C::TILE);
        load_tile<HD>(kv, &tmK, &kv_full[rk.s], kb * AT_T, h, b);
        load_tile<HD>(kv + C::TILE, &tmV, &kv_full[rk.s], kb * AT_T, h, b);
      }
      __syncwarp();
      rk.step();
#pragma unroll 1
      for (int it = 0; it < nit; ++it) {
        const int st = rq.s;
        const int q0 = (qb_first + it) * AT_T;
        if (!mbar_wait_warp(&do_empty[st], rq.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&do_full[st], C::TILE);
          load_tile<HD>(smem + C::OFF_DO + st * C::TILE, &tmDO, &do_full[st], q0, h, b);
        }
        __syncwarp();
        if (!mbar_wait_warp(&q_empty[st], rq.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
        float* sl = stat + st * 256;          // published by the arrive below
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          sl[lane + 32 * u] = -lse_r[u];
          sl[128 + lane + 32 * u] = -dl_r[u];
        }
        __syncwarp();
        if (elect_one()) {
          mbar_arrive_expect_tx(&q_full[st], C::TILE);
          load_tile<HD>(smem + C::OFF_Q + st * C::TILE, &tmQ, &q_full[st], q0, h, b);
        }
        __syncwarp();
        rq.step();
        if (it + 1 < nit) fetch_stats(it + 1);
      }
    }
  } else if (warp == BW_WARP_MMA) {
    // ---------------------------------------------------------- issuer 1: S^T = K Q^T, dP^T = V dO^T
    // (two issuing warps with head_dim 64: the issuing thread runs in step with the tensor pipe, so the waits and
    // descriptor steps of one product would otherwise idle the pipe for the other)
    const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t kv_addr = smem_u32(smem + C::OFF_KV);
    const uint32_t q_addr = smem_u32(smem + C::OFF_Q), do_addr = smem_u32(smem + C::OFF_DO);
    if constexpr (C::TS) {
      Ring<C::STAGES> rq;
      Ring<C::KVB> rk;
      uint32_t ph = 0;             // parity of the previous block
      bool ok = true, first = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const int nit = nq_all - (p.causal ? p.by_hb.div(item) : 0);
        if (!mbar_wait_warp(&kv_full[rk.s], rk.ph, ctx, FT_ERR_WAIT_FULL)) break;
        const uint32_t k_addr = kv_addr + rk.s * 2 * C::TILE, v_addr = k_addr + C::TILE;
#pragma unroll 1
        for (int i = 0; i < nit; ++i) {
          // needs Q_i / dO_i and the score tiles of the previous block copied to registers
          if (!mbar_wait_warp(&do_full[rq.s], rq.ph, ctx, FT_ERR_WAIT_FULL) ||
              !mbar_wait_warp(&q_full[rq.s], rq.ph, ctx, FT_ERR_WAIT_FULL) ||
              (!first && !mbar_wait_warp(st_free, ph, ctx, FT_ERR_WAIT_TMEM_EMPTY))) { ok = false; break; }
          if (!first) ph ^= 1u;
          first = false;
          tc_fence_after();
          if (elect_one()) {
            mma_kmajor<HD>(tmem_base + C::TM_ST, k_addr, q_addr + rq.s * C::TILE, idesc_s);
            mma_kmajor<HD>(tmem_base + C::TM_DPT, v_addr, do_addr + rq.s * C::TILE, idesc_s);
            umma_commit(st_full);
            if (i == nit - 1) umma_commit(&kv_empty[rk.s]);
          }
          __syncwarp();
          rq.step();
        }
        rk.step();
      }
    } else {
      // One issuer for all four products of head_dim 128.  In the steady state block g + 1's dP^T runs under block g's
      // exponentials, then dV += P^T dO as soon as P^T is there, the next scores as soon as dV has read P^T (which lies
      // in their columns), and dK last, under the next exponentials.
      const uint32_t idesc_acc = make_idesc_bf16(128, HD, 0, 1);
      const uint32_t dst_addr = smem_u32(smem + C::OFF_DST);
      const uint32_t k_addr = kv_addr, v_addr = kv_addr + C::TILE;
      Ring<C::STAGES> rn, rc;      // stage of the next block's scores, of the current block
      uint32_t kv_ph = 0, blk = 0, tile_ph = 0;      // parity of the item, of the block, of the finished item
      bool ok = true;
      auto dp_next = [&]() -> bool {
        if (!mbar_wait_warp(&do_full[rn.s], rn.ph, ctx, FT_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        if (elect_one()) mma_kmajor<HD>(tmem_base + C::TM_DPT, v_addr, do_addr + rn.s * C::TILE, idesc_s);
        __syncwarp();
        return true;
      };
      auto s_next = [&](bool last) -> bool {
        if (!mbar_wait_warp(&q_full[rn.s], rn.ph, ctx, FT_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        if (elect_one()) {
          mma_kmajor<HD>(tmem_base + C::TM_ST, k_addr, q_addr + rn.s * C::TILE, idesc_s);
          umma_commit(st_full);
          if (last) umma_commit(&kv_empty[0]);
        }
        __syncwarp();
        rn.step();
        return true;
      };
      bool first_item = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const int nit = nq_all - (p.causal ? p.by_hb.div(item) : 0);
        // the item's first scores (the score columns are free: its predecessor's last dV has finished)
        ok = mbar_wait_warp(&kv_full[0], kv_ph, ctx, FT_ERR_WAIT_FULL) && dp_next() && s_next(nit == 1);
        if (!ok) break;
        kv_ph ^= 1u;
#pragma unroll 1
        for (int i = 0; i < nit; ++i) {
          const bool more = i + 1 < nit;
          if (more && (!mbar_wait_warp(st_free, blk, ctx, FT_ERR_WAIT_TMEM_EMPTY) || !dp_next())) { ok = false; break; }
          if (!mbar_wait_warp(pt_ready, blk, ctx, FT_ERR_WAIT_SOFTMAX) ||
              (i == 0 && !first_item && !mbar_wait_warp(acc_free, tile_ph, ctx, FT_ERR_WAIT_TMEM_EMPTY))) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            mma_ptmem_times_rows(tmem_base + C::TM_DV, tmem_base + C::TM_PT, do_addr + rc.s * C::TILE, idesc_acc, i > 0);
            umma_commit(dv_done);
            umma_commit(&do_empty[rc.s]);
          }
          __syncwarp();
          if (!mbar_wait_warp(dv_done, blk, ctx, FT_ERR_WAIT_TMEM_FULL) || (more && !s_next(i + 2 == nit)) ||
              !mbar_wait_warp(ds_ready, blk, ctx, FT_ERR_WAIT_SOFTMAX)) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            mma_p_times_rows(tmem_base + C::TM_DK, dst_addr, q_addr + rc.s * C::TILE, idesc_acc, i > 0);
            umma_commit(acc_done);
            umma_commit(&q_empty[rc.s]);
          }
          __syncwarp();
          rc.step();
          blk ^= 1u;
        }
        if (!first_item) tile_ph ^= 1u;
        first_item = false;
      }
    }
  } else if (warp == BW_WARP_MMA2) {
    if constexpr (C::TS) {
      // ---------------------------------------------------------- issuer 2: dV += P^T dO, dK += dS^T Q
      const uint32_t idesc_acc = make_idesc_bf16(128, HD, 0, 1);
      const uint32_t q_addr = smem_u32(smem + C::OFF_Q), do_addr = smem_u32(smem + C::OFF_DO);
      Ring<C::STAGES> rq;
      uint32_t blk = 0, tile_ph = 0;
      bool ok = true, first_item = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const int nit = nq_all - (p.causal ? p.by_hb.div(item) : 0);
#pragma unroll 1
        for (int it = 0; it < nit; ++it) {
          if (!mbar_wait_warp(pt_ready, blk, ctx, FT_ERR_WAIT_SOFTMAX) ||
              (it == 0 && !first_item && !mbar_wait_warp(acc_free, tile_ph, ctx, FT_ERR_WAIT_TMEM_EMPTY))) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            mma_ptmem_times_rows(tmem_base + C::TM_DV, tmem_base + C::TM_PT, do_addr + rq.s * C::TILE, idesc_acc, it > 0);
            mma_ptmem_times_rows(tmem_base + C::TM_DK, tmem_base + C::TM_DST, q_addr + rq.s * C::TILE, idesc_acc, it > 0);
            umma_commit(acc_done);
            umma_commit(&do_empty[rq.s]);      // S^T / dP^T of this stage finished before the math ran
            umma_commit(&q_empty[rq.s]);
          }
          __syncwarp();
          rq.step();
          blk ^= 1u;
        }
        if (!first_item) tile_ph ^= 1u;
        first_item = false;
      }
    }
  } else if (warp < BW_MATH) {
    const int g = warp >> 2;               // column group: queries [32 g, 32 g + 32) of the block
    const int qd = warp & 3;
    const int row = qd * 32 + lane;        // key row of this thread
    const int c0 = 32 * g;
    const uint32_t lane_sel = (uint32_t)(qd * 32) << 16;
    const f32x2 sl2 = pk2(p.sl2, p.sl2);
    Ring<C::STAGES> rq;
    uint32_t blk = 0;                      // parity of the block
    bool ok = true, first = true;
    uint8_t* box = smem + C::OFF_DST + warp * BW_BOX;
    // dV and dK of a finished item: 2 HD / 32 column chunks (dV first) spread over the four groups
    auto drain = [&](int kb, int b, int h) {
      constexpr int NCH = 2 * HD / 32 / 4;
      tc_fence_after();
      uint32_t r[NCH][32];
#pragma unroll
      for (int u = 0; u < NCH; ++u) tmem_ld32(tmem_base + C::TM_DV + (g + 4 * u) * 32 + lane_sel, r[u]);
      tmem_ld_wait();
      tc_fence_before();
      if (C::TS && lane == 0) bulk_wait_read_all();      // the box of the item before
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
#pragma unroll
      for (int u = 0; u < NCH; ++u) {
        const int ch = g + 4 * u;
        const bool is_dk = ch >= HD / 32;
        if (u > 0) {
          if (lane == 0) bulk_wait_read_all();
          __syncwarp();
        }
        store_out32(box, lane, r[u], is_dk ? p.scale : 1.f, &out.m[is_dk ? 1 : 0], (is_dk ? ch - HD / 32 : ch) * 32,
                    kb * AT_T + qd * 32, h, b, p.S);
      }
    };
    // LATE (head_dim 64): an item's output leaves behind the first block of the next item, so the exponentials wait neither for its
    // last products nor for the drain (between two items' blocks went ~3300 cycles, 800 of them for the products and 2100 for the
    // output, where a block takes 1830: B8 S1024 H12 causal, five items a CTA, 45.7 -> 39.7 us).  head_dim 128: it is staged in
    // the dS^T tile and leaves at once (B4 S2048 H16 149 -> 142 us by the TMA stores alone).
    int late_kb = -1, late_b = 0, late_h = 0;
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const int kb = p.by_hb.div(item), hb = item - kb * n_hb, b = p.by_h.div(hb), h = hb - b * p.H;
      const int k0 = kb * AT_T, gk = k0 + row;
      const int qb_first = p.causal ? kb : 0, nit = nq_all - qb_first;
#pragma unroll 1
      for (int it = 0; it < nit; ++it) {
        const int st = rq.s;
        const int q0 = (qb_first + it) * AT_T;
        // statistics were written by the producer before its arrive on q_full
        if (!mbar_wait_warp(&q_full[st], rq.ph, ctx, FT_ERR_WAIT_FULL) ||
            !mbar_wait_warp(st_full, blk, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
        uint32_t rs[32], rd[32];
        tmem_ld32(tmem_base + C::TM_ST + c0 + lane_sel, rs);
        tmem_ld32(tmem_base + C::TM_DPT + c0 + lane_sel, rd);
        tmem_ld_wait();
        tc_fence_before();
        // (head_dim 128: behind st_free every warp's output has left the dS^T tile)
        if (!C::TS && it == 0 && lane == 0) bulk_wait_read_all();
        __syncwarp();
        if (lane == 0) mbar_arrive(st_free);      // one arrival per warp
        const float4* sl4 = reinterpret_cast<const float4*>(stat + st * 256 + c0);
        const float4* dl4 = reinterpret_cast<const float4*>(stat + st * 256 + 128 + c0);
        // Queries before the key become -inf, in the diagonal block and the warps that hold such pairs only.  Queries past
        // the end have -lse = -inf; key rows past the end are never stored and touch no other row.
        if (p.causal && q0 + c0 < k0 + qd * 32 + 31) {
          const int lo = gk - q0 - c0;            // first valid column of this thread
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < lo) rs[i] = __float_as_uint(-INFINITY);
        }
        uint32_t pw[16], dw[16];
        if constexpr (C::TS) {
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            const float4 nl = sl4[i4], dl = dl4[i4];
            const f32x2 e0 = exp2_pair(fma2(acc2(rs, 4 * i4), sl2, pk2(nl.x, nl.y)));
            const f32x2 e1 = exp2_pair(fma2(acc2(rs, 4 * i4 + 2), sl2, pk2(nl.z, nl.w)));
            pw[2 * i4] = pack2(e0);
            pw[2 * i4 + 1] = pack2(e1);
            dw[2 * i4] = pack2(mul2(e0, add2(acc2(rd, 4 * i4), pk2(dl.x, dl.y))));
            dw[2 * i4 + 1] = pack2(mul2(e1, add2(acc2(rd, 4 * i4 + 2), pk2(dl.z, dl.w))));
          }
          // the operand tiles' previous readers (dV / dK of the block before) must have finished
          if (!first && !mbar_wait_warp(acc_done, blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
          // this thread's 32 queries of its key row: 16 packed columns of each operand tile
          tc_fence_after();
          tmem_st16(tmem_base + C::TM_PT + 16 * g + lane_sel, pw);
          tmem_st16(tmem_base + C::TM_DST + 16 * g + lane_sel, dw);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(pt_ready);      // one arrival per warp
          if (LATE && late_kb >= 0) {                // (acc_done of its last block was waited for above)
            drain(late_kb, late_b, late_h);
            late_kb = -1;
          }
        } else {
          f32x2 e[16];
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            const float4 nl = sl4[i4];
            e[2 * i4] = exp2_pair(fma2(acc2(rs, 4 * i4), sl2, pk2(nl.x, nl.y)));
            e[2 * i4 + 1] = exp2_pair(fma2(acc2(rs, 4 * i4 + 2), sl2, pk2(nl.z, nl.w)));
            pw[2 * i4] = pack2(e[2 * i4]);
            pw[2 * i4 + 1] = pack2(e[2 * i4 + 1]);
          }
          // P^T goes where the scores were, once every warp has copied its part of them
          if (!mbar_wait_warp(st_free, blk, ctx, FT_ERR_WAIT_WARPS)) { ok = false; break; }
          tc_fence_after();
          tmem_st16(tmem_base + C::TM_PT + 16 * g + lane_sel, pw);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(pt_ready);
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            const float4 dl = dl4[i4];
            dw[2 * i4] = pack2(mul2(e[2 * i4], add2(acc2(rd, 4 * i4), pk2(dl.x, dl.y))));
            dw[2 * i4 + 1] = pack2(mul2(e[2 * i4 + 1], add2(acc2(rd, 4 * i4 + 2), pk2(dl.z, dl.w))));
          }
          if (!first && !mbar_wait_warp(acc_done, blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
          store_row32_packed(smem + C::OFF_DST, row, c0, dw);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(ds_ready);
        }
        first = false;
        rq.step();
        blk ^= 1u;
      }
      if (!ok) break;
      if (LATE) {
        late_kb = kb;
        late_b = b;
        late_h = h;
        continue;
      }
      if (!mbar_wait_warp(acc_done, blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      drain(kb, b, h);
    }
    if (LATE && ok && late_kb >= 0 && mbar_wait_warp(acc_done, blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) drain(late_kb, late_b, late_h);
    if (lane == 0) bulk_wait_read_all();
  }

  if (*abort_f) {
    for (int i = 0; i < 100; ++i) __nanosleep(10000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == BW_WARP_MMA) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// =============================================================================== backward: dQ
template <int HD>
struct DqCfg {
  static constexpr int TILE = (HD / 64) * AT_REGION;
  static constexpr int QB = (HD == 64) ? 2 : 1;          // Q / dO buffers (one per work item)
  // K and V have a ring each: a V tile is free after dP, a K tile only after dQ, most of two blocks later.  (In one ring of
  // four tiles the load of every second K started when it was needed: 2000 cycles per pair of blocks.  B4 S2048 H16 causal, head
  // size 128: 126 -> 110 us.)
  static constexpr int KS = (HD == 64) ? 4 : 3;
  static constexpr int VS = (HD == 64) ? 4 : 2;
  static constexpr int OFF_QDO = 0;                      // [QB] Q, dO
  static constexpr int OFF_K = QB * 2 * TILE;            // [KS]; an item's output leaves through its last one
  static constexpr int OFF_V = OFF_K + KS * TILE;        // [VS]
  static constexpr int OFF_BAR = OFF_V + VS * TILE;
  static constexpr int OFF_DELTA = OFF_BAR + 512;        // [2] rowsum(dO o O) of an item's rows
  static constexpr int SMEM = OFF_DELTA + 2 * AT_T * 4;
  // rowsum(dO o O): LPR lanes share a row, each of the 16 math warps takes 8 rows in U steps
  static constexpr int LPR = HD / 8, RPS = 32 / LPR, U = 8 / RPS;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0, TM_DP = 128, TM_DQ = 256;
  static constexpr int TM_DS = 384;                      // dS buffer i (packed bf16) at TM_DS + 64 i
  static_assert(SMEM <= 232448, "shared memory");
};

// Persistent like the dK / dV kernel.  dS goes to the tensor core through tensor memory, two buffers.  Between two items (MANY: some
// CTA has a second one): the Q and dO tiles go back to the loader with the last score products, delta of the next item is made
// under the last dQ product, and the output leaves through the K tile of the last block, which the loader gets back when it has
// left.  (Staged in the Q tile, with one such buffer for head_dim 128, an item waited ~2500 cycles for its tiles and made delta
// behind them: B4 S2048 H16 causal 111 -> 101 us, B8 S1024 H12 head size 64 43.2 -> 40.6 us.)
//
// It also makes delta = rowsum(dO o O), which the dK / dV kernel behind it reads: dO is in shared memory here anyway and the
// item's share of O is fetched one item ahead.  (A kernel of its own
// in front of both read dO once more and stood on the path of the whole backward: B8 S1024 H12 head size 64 causal 75.1 -> 72.5 us,
// B4 S2048 H16 head size 128 252 -> 246 us, B4 S128 H2 11.7 -> 10.4 us.)
template <int HD, bool MANY>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmDQ, const AttnArgs p) {
  using C = DqCfg<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* qdo_full = bars;        // [2]
  uint64_t* qdo_empty = bars + 2;   // [2] the item's score products are done, its delta is made (one arrival per warp)
  uint64_t* k_full = bars + 4;      // [4]
  uint64_t* k_empty = bars + 8;     // [4]
  uint64_t* v_full = bars + 12;     // [4]
  uint64_t* v_empty = bars + 16;    // [4]
  uint64_t* s_full = bars + 20;     // S and dP in TMEM
  uint64_t* s_free = bars + 21;     // both copied to registers (one arrival per warp)
  uint64_t* ds_ready = bars + 22;   // [2] dS handed to the tensor core (one arrival per warp)
  uint64_t* acc_done = bars + 24;   // [2] dQ product that read the buffer done
  uint64_t* acc_free = bars + 26;   // the item's dQ copied to registers (one arrival per warp)
  uint64_t* d_ready = bars + 27;    // the item's delta is in shared memory (one arrival per warp)
  uint64_t* out_done = bars + 28;   // [4] the output that went through the K tile has left it (one arrival per warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
  int* abort_f = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  WaitCtx ctx{p.status, abort_f};

  if ((smem_u32(smem) & 1023u) != 0u) {
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(p.status, 0, FT_ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&out_done[i], BW_MATH);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&qdo_full[i], 1);
      mbar_init(&qdo_empty[i], BW_MATH + 1);
      mbar_init(&ds_ready[i], BW_MATH);
      mbar_init(&acc_done[i], 1);
    }
    for (int i = 0; i < 16; ++i) mbar_init(&k_full[i], 1);      // the four arrays of the rings
    mbar_init(s_full, 1);
    mbar_init(s_free, BW_MATH);
    mbar_init(acc_free, BW_MATH);
    mbar_init(d_ready, BW_MATH);
    *abort_f = 0;
    fence_mbar_init();
  }
  if (warp == BW_WARP_TMA && elect_one()) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == BW_WARP_MMA) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  // items are numbered with the most key blocks (the late query blocks under a causal mask) first
  const int n_hb = p.H * p.B;
  const int nkv_all = (p.S + AT_T - 1) / AT_T;
  auto query_block = [&](int item) { return nkv_all - 1 - p.by_hb.div(item); };
  auto key_blocks = [&](int qb) { return p.causal ? qb + 1 : nkv_all; };
  TileWalk walk(p.n_tiles);

  if (warp == BW_WARP_TMA) {
    Ring<C::QB> rq;
    Ring<C::KS> rk;
    Ring<C::VS> rv;
    bool ok = true;
    uint32_t staged = 0, staged_ph = 0;      // K tiles that an output goes through, parities of out_done
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const int qb = query_block(item), hb = item - (nkv_all - 1 - qb) * n_hb, b = p.by_h.div(hb), h = hb - b * p.H;
      const int nkv = key_blocks(qb);
      if (!mbar_wait_warp(&qdo_empty[rq.s], rq.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) break;
      if (elect_one()) {
        uint8_t* qd = smem + C::OFF_QDO + rq.s * 2 * C::TILE;
        mbar_arrive_expect_tx(&qdo_full[rq.s], 2 * C::TILE);
        load_tile<HD>(qd, &tmQ, &qdo_full[rq.s], qb * AT_T, h, b);
        load_tile<HD>(qd + C::TILE, &tmDO, &qdo_full[rq.s], qb * AT_T, h, b);
      }
      __syncwarp();
      rq.step();
#pragma unroll 1
      for (int j = 0; j < nkv; ++j) {
        if (!mbar_wait_warp(&k_empty[rk.s], rk.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
        if ((staged >> rk.s) & 1u) {
          if (!mbar_wait_warp(&out_done[rk.s], (staged_ph >> rk.s) & 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
          staged &= ~(1u << rk.s);
          staged_ph ^= 1u << rk.s;
        }
        if (j == nkv - 1) staged |= 1u << rk.s;
        if (elect_one()) {
          mbar_arrive_expect_tx(&k_full[rk.s], C::TILE);
          load_tile<HD>(smem + C::OFF_K + rk.s * C::TILE, &tmK, &k_full[rk.s], j * AT_T, h, b);
        }
        __syncwarp();
        rk.step();
        if (!mbar_wait_warp(&v_empty[rv.s], rv.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&v_full[rv.s], C::TILE);
          load_tile<HD>(smem + C::OFF_V + rv.s * C::TILE, &tmV, &v_full[rv.s], j * AT_T, h, b);
        }
        __syncwarp();
        rv.step();
      }
    }
  } else if (warp == BW_WARP_MMA) {
    // ---------------------------------------------------------- issuer 1: S = Q K^T, dP = dO V^T
    const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t qdo_addr = smem_u32(smem + C::OFF_QDO);
    const uint32_t k_addr = smem_u32(smem + C::OFF_K), v_addr = smem_u32(smem + C::OFF_V);
    Ring<C::QB> rq;
    Ring<C::KS> rk;
    Ring<C::VS> rv;
    uint32_t ph = 0;
    bool ok = true, first = true;
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const int nkv = key_blocks(query_block(item));
      if (!mbar_wait_warp(&qdo_full[rq.s], rq.ph, ctx, FT_ERR_WAIT_FULL)) break;
      const uint32_t q_addr = qdo_addr + rq.s * 2 * C::TILE, do_addr = q_addr + C::TILE;
#pragma unroll 1
      for (int j = 0; j < nkv; ++j) {
        if (!mbar_wait_warp(&k_full[rk.s], rk.ph, ctx, FT_ERR_WAIT_FULL) ||
            (!first && !mbar_wait_warp(s_free, ph, ctx, FT_ERR_WAIT_TMEM_EMPTY))) { ok = false; break; }
        if (!first) ph ^= 1u;
        first = false;
        tc_fence_after();
        if (elect_one()) mma_kmajor<HD>(tmem_base + C::TM_S, q_addr, k_addr + rk.s * C::TILE, idesc_s);
        __syncwarp();
        rk.step();
        if (!mbar_wait_warp(&v_full[rv.s], rv.ph, ctx, FT_ERR_WAIT_FULL)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          mma_kmajor<HD>(tmem_base + C::TM_DP, do_addr, v_addr + rv.s * C::TILE, idesc_s);
          umma_commit(s_full);
          umma_commit(&v_empty[rv.s]);
          if (j == nkv - 1) umma_commit(&qdo_empty[rq.s]);
        }
        __syncwarp();
        rv.step();
      }
      rq.step();
    }
  } else if (warp == BW_WARP_MMA2) {
    // ---------------------------------------------------------- issuer 2: dQ += dS K
    const uint32_t idesc_acc = make_idesc_bf16(128, HD, 0, 1);
    const uint32_t k_addr = smem_u32(smem + C::OFF_K);
    Ring<C::KS> rk;
    Ring<2> rd;
    uint32_t tile_ph = 0;
    bool ok = true, first_item = true;
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const int nkv = key_blocks(query_block(item));
#pragma unroll 1
      for (int j = 0; j < nkv; ++j) {
        // (K_j landed before the scores that dS_j was made from)
        if (!mbar_wait_warp(&ds_ready[rd.s], rd.ph, ctx, FT_ERR_WAIT_SOFTMAX) ||
            (j == 0 && !first_item && !mbar_wait_warp(acc_free, tile_ph, ctx, FT_ERR_WAIT_TMEM_EMPTY))) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          mma_ptmem_times_rows(tmem_base + C::TM_DQ, tmem_base + C::TM_DS + 64 * rd.s, k_addr + rk.s * C::TILE,
                               idesc_acc, j > 0);
          umma_commit(&acc_done[rd.s]);
          umma_commit(&k_empty[rk.s]);       // S of this tile finished before the math ran
        }
        __syncwarp();
        rk.step();
        rd.step();
      }
      if (!first_item) tile_ph ^= 1u;
      first_item = false;
    }
  } else if (warp < BW_MATH) {
    const int g = warp >> 2;               // column group: keys [32 g, 32 g + 32) of the block
    const int qd = warp & 3;
    const int row = qd * 32 + lane;
    const int c0 = 32 * g;
    const uint32_t lane_sel = (uint32_t)(qd * 32) << 16;
    const f32x2 sl2 = pk2(p.sl2, p.sl2);
    Ring<2> rd;
    uint32_t blk = 0;                      // parity of the block
    int filled = 0;                        // dS buffers written so far (2 = both have had a reader)
    bool ok = true;
    // log-sum-exp of this thread's row and this lane's segments of O, fetched one item ahead (used, and signs changed, then)
    float lse_n = 0.f;
    uint4 o_n[C::U];
    const int d_row = 8 * warp + lane / C::LPR, d_seg = lane % C::LPR;      // row of step 0, 16-byte segment
    float* s_delta = reinterpret_cast<float*>(smem + C::OFF_DELTA);
    uint32_t it_ph = 0;                    // parity of the item: d_ready's phase and the buffer of s_delta
    auto fetch_rows = [&](int item) {
      if (item < 0) return;
      const int qb = query_block(item), hb = item - (nkv_all - 1 - qb) * n_hb, b = p.by_h.div(hb), h = hb - b * p.H;
      const int q0 = qb * AT_T;
      lse_n = INFINITY;
      if (q0 + row < p.S) lse_n = p.lse[(long long)hb * p.S + q0 + row];      // [B, H, S]
      const __nv_bfloat16* op = p.o + b * p.o_bs + (long long)(q0 + d_row) * p.o_ss + h * p.o_hs + d_seg * 8;
#pragma unroll
      for (int u = 0; u < C::U; ++u) {
        o_n[u] = make_uint4(0u, 0u, 0u, 0u);
        if (q0 + d_row + u * C::RPS < p.S) o_n[u] = *reinterpret_cast<const uint4*>(op + (long long)(u * C::RPS) * p.o_ss);
      }
    };
    Ring<C::QB> rq;
    Ring<C::KS> rk;
    // delta of an item, from its dO tile and the rows that were fetched
    auto make_delta = [&](int item, uint32_t buf) -> bool {
      const int qb = query_block(item), hb = item - (nkv_all - 1 - qb) * n_hb, q0 = qb * AT_T;
      if (!mbar_wait_warp(&qdo_full[rq.s], rq.ph, ctx, FT_ERR_WAIT_FULL)) return false;
      const uint8_t* do_tile = smem + C::OFF_QDO + (rq.s * 2 + 1) * C::TILE + (d_seg >> 3) * AT_REGION;
      float* s_dl = s_delta + buf * AT_T;
#pragma unroll
      for (int u = 0; u < C::U; ++u) {
        const int r = d_row + u * C::RPS;
        const uint4 g = *reinterpret_cast<const uint4*>(do_tile + r * 128 + (((d_seg & 7) ^ (r & 7)) << 4));
        const uint32_t ow[4] = {o_n[u].x, o_n[u].y, o_n[u].z, o_n[u].w}, gw[4] = {g.x, g.y, g.z, g.w};
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = unpack_bf16(ow[i]), y = unpack_bf16(gw[i]);
          acc = fmaf(x.x, y.x, acc);
          acc = fmaf(x.y, y.y, acc);
        }
#pragma unroll
        for (int m = C::LPR / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
        if (d_seg == 0) {
          s_dl[r] = acc;
          if (q0 + r < p.S) p.delta[(long long)hb * p.S + q0 + r] = acc;
        }
      }
      fence_proxy_async_smem();      // the dO tile goes back to the loader
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(d_ready);
        mbar_arrive(&qdo_empty[rq.s]);
      }
      rq.step();
      return true;
    };
    int item = walk.next();
    fetch_rows(item);
    ok = item >= 0 && make_delta(item, 0);
    int staged = -1;                       // K tile that this warp's last output has not yet left
    auto output_left = [&] {
      if (staged >= 0 && lane == 0) {
        bulk_wait_read_all();
        mbar_arrive(&out_done[staged]);
      }
      staged = -1;
    };
    while (ok && item >= 0) {
      const int qb = query_block(item), hb = item - (nkv_all - 1 - qb) * n_hb, b = p.by_h.div(hb), h = hb - b * p.H;
      const int q0 = qb * AT_T, grow = q0 + row, nkv = key_blocks(qb);
      const f32x2 nl = pk2(-lse_n, -lse_n);
      item = MANY ? walk.next() : -1;
      if (MANY) fetch_rows(item);
      if (!mbar_wait_warp(d_ready, it_ph, ctx, FT_ERR_WAIT_WARPS)) { ok = false; break; }
      const float dl_row = -s_delta[it_ph * AT_T + row];
      it_ph ^= 1u;
      const f32x2 dl = pk2(dl_row, dl_row);
      const int last_col = p.causal ? min(grow, p.S - 1) : p.S - 1;                 // last valid key of this row
      const int warp_last = p.causal ? min(q0 + qd * 32, p.S - 1) : p.S - 1;       // of the warp's first row
#pragma unroll 1
      for (int j = 0; j < nkv; ++j) {
        if (!mbar_wait_warp(s_full, blk, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
        uint32_t rs[32], rdp[32];
        tmem_ld32(tmem_base + C::TM_S + c0 + lane_sel, rs);
        tmem_ld32(tmem_base + C::TM_DP + c0 + lane_sel, rdp);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);      // one arrival per warp
        const int k0 = j * AT_T + c0;
        uint32_t dw[16];
        if (k0 + 31 > warp_last) {      // masked scores become -inf in a pass of their own
          const int lim = last_col - k0;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i > lim) rs[i] = __float_as_uint(-INFINITY);
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const f32x2 e = exp2_pair(fma2(acc2(rs, i), sl2, nl));
          dw[i >> 1] = pack2(mul2(e, add2(acc2(rdp, i), dl)));
        }
        if (filled == 2 && !mbar_wait_warp(&acc_done[rd.s], rd.ph ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
        if (filled < 2) ++filled;
        tc_fence_after();
        tmem_st16(tmem_base + C::TM_DS + 64 * rd.s + 16 * g + lane_sel, dw);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_ready[rd.s]);      // one arrival per warp
        rd.step();
        blk ^= 1u;
        if (MANY && j == 0) output_left();
        if (j + 1 < nkv) rk.step();
      }
      // under the last product: delta of the next item (whose tiles were loaded under the last block)
      if (MANY && ok && item >= 0) ok = make_delta(item, it_ph);
      // the buffer of the last block is the one before rd
      if (!ok || !mbar_wait_warp(&acc_done[rd.s ^ 1], rd.s == 0 ? rd.ph ^ 1u : rd.ph, ctx, FT_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (g < HD / 32) {
        uint32_t r[32];
        tmem_ld32(tmem_base + C::TM_DQ + g * 32 + lane_sel, r);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_free);
        store_out32(smem + C::OFF_K + rk.s * C::TILE + warp * BW_BOX, lane, r, p.scale, &tmDQ, c0, q0 + qd * 32, h, b, p.S);
      } else if (lane == 0) {
        mbar_arrive(acc_free);
      }
      staged = rk.s;
      rk.step();
    }
    output_left();
  }

  if (*abort_f) {
    for (int i = 0; i < 100; ++i) __nanosleep(10000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == BW_WARP_MMA) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

template <int HD>
static int attn_bwd_launch(const FtkAttnDesc* a, cudaStream_t s) {
  CUtensorMap tq, tk, tv, tdo, tdq;
  DkvMaps out;
  int rc;
  if ((rc = make_map(&tq, a->q, a, a->q_bs, a->q_ss, a->q_hs))) return rc;
  if ((rc = make_map(&tk, a->k, a, a->k_bs, a->k_ss, a->k_hs))) return rc;
  if ((rc = make_map(&tv, a->v, a, a->v_bs, a->v_ss, a->v_hs))) return rc;
  if ((rc = make_map(&tdo, a->d_o, a, a->o_bs, a->o_ss, a->o_hs))) return rc;
  if ((rc = make_map(&tdq, a->dq, a, a->q_bs, a->q_ss, a->q_hs, 32, 32))) return rc;
  if ((rc = make_map(&out.m[1], a->dk, a, a->k_bs, a->k_ss, a->k_hs, 32, 32))) return rc;
  if ((rc = make_map(&out.m[0], a->dv, a, a->v_bs, a->v_ss, a->v_hs, 32, 32))) return rc;
  AttnArgs p{};
  fill_args(p, a);
  if (!p.status) return -6;
  static bool attr = false;
  if (!attr) {
    if ((rc = set_smem(attn_bwd_dkv_kernel<HD, false>, DkvCfg<HD>::SMEM))) return rc;
    if ((rc = set_smem(attn_bwd_dkv_kernel<HD, HD == 64>, DkvCfg<HD>::SMEM))) return rc;
    if ((rc = set_smem(attn_bwd_dq_kernel<HD, true>, DqCfg<HD>::SMEM))) return rc;
    if ((rc = set_smem(attn_bwd_dq_kernel<HD, false>, DqCfg<HD>::SMEM))) return rc;
    attr = true;
  }
  const long long nrows = (long long)a->B * a->S * a->H;
  if (nrows > 0x7fffffffll) return -2;
  unsigned grid = 0;
  if ((rc = set_items(p, a, AT_T, &grid))) return rc;
  // An item that ends under the next one costs its kernel's block loop registers: about 70 cycles of 1830 a block.  So where no CTA
  // has a second item both kernels take the form without, and dK / dV ends an item at once also where 1100 cycles saved per item
  // boundary are less than that (blocks per item: half of them under a causal mask).  us, always under the next / by this rule:
  // B1 S4096 H4 causal 62.9 / 60.7, B1 S1024 H12 21.7 / 20.6, B8 S763 H3 20.1 / 19.1 (one item a CTA); B2 S1024 H12 causal 23.5 / 23.1,
  // B1 S4096 H6 causal 65.3 / 64.3; ended at once / by this rule: B8 S256 H12 15.8 / 15.0, B4 S1024 H12 37.2 / 36.3.
  const long long items = p.n_tiles, nb = (a->S + AT_T - 1) / AT_T;
  const bool many = items > (long long)grid;
  const bool late = HD == 64 && 32 * (items - (long long)grid) > items * (a->causal ? nb + 1 : 2 * nb);
  auto dq = many ? attn_bwd_dq_kernel<HD, true> : attn_bwd_dq_kernel<HD, false>;
  auto dkv = late ? attn_bwd_dkv_kernel<HD, HD == 64> : attn_bwd_dkv_kernel<HD, false>;
  launch_pdl(dq, grid, BW_THREADS, DqCfg<HD>::SMEM, s, tq, tk, tv, tdo, tdq, p);      // writes delta
  launch_pdl(dkv, grid, BW_THREADS, DkvCfg<HD>::SMEM, s, tq, tk, tv, tdo, out, p);
  return (int)cudaGetLastError();
}

}  // namespace ftk

using namespace ftk;

extern "C" int ftk_attn_bwd(const FtkAttnDesc* a, void* stream) {
  if (!a || a->B <= 0 || a->H <= 0 || a->S <= 0 || !a->delta || !a->lse) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a->hd == 64) return attn_bwd_launch<64>(a, s);
  if (a->hd == 128) return attn_bwd_launch<128>(a, s);
  return -5;
}
