// Flash attention forward for sm_100a (tcgen05 / TMEM), head_dim 64 or 128.
//
// Semantics: ft-kernel-cpu/src/lib.rs:4572 sdpa_forward_f64 (blockwise QK^T -> stable online
// softmax -> PV, causal masks j > i); block-online rescaling as in the Metal attn_flash2
// shader (ft-kernel-metal/src/fused.rs:407).  Output O (bf16) and the log-sum-exp in the
// log2 domain of the scaled scores (fp32 [B, H, S]) for the recompute backward.
//
// One persistent CTA per SM walks items of 256 query rows (two 128-row tiles) of one (batch, head) and streams K and V
// blocks of 128 keys through two TMA rings (a ring per role that waits on it: with one ring of an odd number of slots for
// both, the issuer of the scores could take the landing of a slot's V tile for that of the K tile after it).  Rings, barriers
// and tile buffers run on across items, so an item's loads and first scores are issued under the output of the one
// before.  12 warps:
//   warps 0-3  softmax group A (tile 0), warps 4-7 softmax group B (tile 1): one thread per
//              query row reads its whole 128-wide score row into registers with tcgen05.ld;
//   warp 8     TMA producer;  warp 9  issues S = Q K^T (owns TMEM);  warp 10 issues O += P V;
//              warp 11 only hands its registers to the softmax groups (setmaxnreg).
// The output accumulates in TMEM across all key blocks.  The running maximum is lazy: a row
// keeps its reference maximum until a block exceeds it by more than 2^8, and only then is the
// TMEM accumulator rescaled (tcgen05.ld / mul / tcgen05.st, voted per warp).  The probabilities stay in tensor memory
// (tcgen05.st of packed bf16 pairs by the row's thread) and P V is issued with its A operand there.  With head_dim 64 they
// have columns of their own and QK^T of the next block runs under the exponentials of this one; with head_dim 128 all 512
// columns are taken by S and O, so P overwrites the scores it was made from and a tile's next scores follow its P V - the
// two tiles take turns on the tensor core and on the exponentials.
#include "attn_common.cuh"
#include "attn_turns.h"

namespace ftk {

constexpr int F2_THREADS = 384;
constexpr float F2_LAZY = 8.0f;       // log2 headroom before the accumulator is rescaled

template <int HD>
struct Fwd2Cfg {
  static constexpr int TILE = (HD / 64) * AT_REGION;        // one [128 x HD] bf16 tile
  static constexpr bool ALIAS = (HD == 128);                // P in the columns of S
  static constexpr bool TURNS = !ALIAS;                     // the groups' exponentials alternate
  static constexpr int QS = (HD == 64) ? 4 : 3;             // Q tiles
  static constexpr int KS = (HD == 64) ? 4 : 2;             // K ring
  static constexpr int VS = (HD == 64) ? 4 : 2;             // V ring
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + QS * TILE;
  static constexpr int OFF_V = OFF_K + KS * TILE;
  static constexpr int OFF_BAR = OFF_V + VS * TILE;
  static constexpr int SMEM = OFF_BAR + 512;
  static constexpr int TMEM_COLS = 512;
  static constexpr int TM_S = 0;                            // S tile t at TM_S + 128 t
  static constexpr int TM_O = 256;                          // O tile t at TM_O + HD t
  static constexpr int TM_P = ALIAS ? TM_S : 256 + 2 * HD;  // P tile t at TM_P + P_STRIDE t
  static constexpr int P_STRIDE = ALIAS ? 128 : 64;
  static_assert(SMEM <= 232448, "shared memory");
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
template <int REGS>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
}
template <int REGS>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
}

// One work item: 256 query rows of one (batch, head).
struct FwdItem {
  int h, b, q0, nb[2], nkv;       // key blocks of each tile (0: no row of the tile exists), of the item
  __device__ __forceinline__ FwdItem(int item, const AttnArgs& p) {
    // items are numbered with the late query blocks (the ones with the most key blocks under a causal mask) first
    const int n_hb = p.H * p.B, n_qb = (p.S + 2 * AT_T - 1) / (2 * AT_T), nkv_all = (p.S + AT_T - 1) / AT_T;
    const int blk = p.by_hb.div(item), hb = item - blk * n_hb;
    b = p.by_h.div(hb);
    h = hb - b * p.H;
    const int qb = n_qb - 1 - blk;
    q0 = qb * 2 * AT_T;
#pragma unroll
    for (int t = 0; t < 2; ++t)
      nb[t] = 2 * qb + t >= nkv_all ? 0 : (p.causal ? 2 * qb + t + 1 : nkv_all);
    nkv = max(nb[0], nb[1]);
  }
};

template <int HD>
__global__ void __launch_bounds__(F2_THREADS, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const AttnArgs p) {
  using C = Fwd2Cfg<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* q_full = bars;             // [4]
  uint64_t* q_empty = bars + 4;        // [4] the item's output has left through the tile (one arrival per warp)
  uint64_t* k_full = bars + 8;         // [4]
  uint64_t* k_empty = bars + 12;       // [4]
  uint64_t* v_full = bars + 16;        // [4]
  uint64_t* v_empty = bars + 20;       // [4]
  uint64_t* s_full = bars + 24;        // [2] per tile: scores in TMEM
  uint64_t* s_free = bars + 26;        // [2] per tile: scores copied to registers (one arrival per warp; not ALIAS)
  uint64_t* p_ready = bars + 28;       // [2][2] per half and tile: probabilities in TMEM (one arrival per warp)
  uint64_t* pv_done = bars + 32;       // [2] per tile: PV finished (P free, O tile settled)
  uint64_t* o_free = bars + 34;        // [2] per tile: the item's O copied to registers (one arrival per warp)
  uint64_t* e_done = bars + 36;        // [2] per tile: the group's turn is over (one arrival per warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 38);
  int* abort_f = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  WaitCtx ctx{p.status, abort_f};

  if ((smem_u32(smem) & 1023u) != 0u) {
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(p.status, 0, FT_ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 24; ++i) mbar_init(&bars[i], i >= 4 && i < 8 ? 4 : 1);    // q_empty: one arrival per warp
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);      // one arrival per warp of the group
      mbar_init(&p_ready[i], 4);
      mbar_init(&p_ready[2 + i], 4);
      mbar_init(&e_done[i], 4);
      mbar_init(&pv_done[i], 1);
      mbar_init(&o_free[i], 4);
    }
    *abort_f = 0;
    fence_mbar_init();
  }
  if (warp == 8 && elect_one()) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();
  TileWalk walk(p.n_tiles);

  if (warp >= 8) {
    reg_dec<40>();
    if (warp == 8) {
      // ------------------------------------------------------------ TMA producer
      Ring<C::QS> rq;
      Ring<C::KS> rk;
      Ring<C::VS> rv;
      bool ok = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const FwdItem it(item, p);
#pragma unroll 1
        for (int j = 0; ok && j < it.nkv; ++j) {
#pragma unroll 1
          for (int t = 0; j == 0 && t < 2; ++t) {
            if (it.nb[t] == 0) continue;
            if (!mbar_wait_warp(&q_empty[rq.s], rq.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
            if (elect_one()) {
              mbar_arrive_expect_tx(&q_full[rq.s], C::TILE);
              load_tile<HD>(smem + C::OFF_Q + rq.s * C::TILE, &tmQ, &q_full[rq.s], it.q0 + t * AT_T, it.h, it.b);
            }
            __syncwarp();
            rq.step();
          }
          if (!ok || !mbar_wait_warp(&k_empty[rk.s], rk.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
          if (elect_one()) {
            mbar_arrive_expect_tx(&k_full[rk.s], C::TILE);
            load_tile<HD>(smem + C::OFF_K + rk.s * C::TILE, &tmK, &k_full[rk.s], j * AT_T, it.h, it.b);
          }
          __syncwarp();
          rk.step();
          if (!mbar_wait_warp(&v_empty[rv.s], rv.ph ^ 1u, ctx, FT_ERR_WAIT_EMPTY)) { ok = false; break; }
          if (elect_one()) {
            mbar_arrive_expect_tx(&v_full[rv.s], C::TILE);
            load_tile<HD>(smem + C::OFF_V + rv.s * C::TILE, &tmV, &v_full[rv.s], j * AT_T, it.h, it.b);
          }
          __syncwarp();
          rv.step();
        }
      }
    } else if (warp == 9) {
      // ------------------------------------------------------------ MMA issuer 1: S = Q K^T
      // The issuing thread runs in step with the tensor pipe (an MMA is accepted when the one
      // before the previous has finished), so every wait, fence and descriptor step between
      // two MMAs is time the pipe idles.  Two issuers, one per product, overlap that overhead.
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t q_addr = smem_u32(smem + C::OFF_Q), k_addr = smem_u32(smem + C::OFF_K);
      Ring<C::QS> rq;
      Ring<C::KS> rk;
      uint32_t seen = 0, blk = 0;        // bit t: a block of tile t has been issued; parity of the last one
      bool ok = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const FwdItem it(item, p);
        uint32_t q_slot[2] = {0, 0};
#pragma unroll 1
        for (int j = 0; ok && j < it.nkv; ++j) {
          if (!mbar_wait_warp(&k_full[rk.s], rk.ph, ctx, FT_ERR_WAIT_FULL)) { ok = false; break; }
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!ok || j >= it.nb[t]) continue;
            if (j == 0) {
              if (!mbar_wait_warp(&q_full[rq.s], rq.ph, ctx, FT_ERR_WAIT_FULL)) { ok = false; continue; }
              q_slot[t] = rq.s;
              rq.step();
            }
            // the tile's previous scores must have been copied to registers (ALIAS: and their P used)
            if (((seen >> t) & 1u) &&
                !mbar_wait_warp(C::ALIAS ? &pv_done[t] : &s_free[t], (blk >> t) & 1u, ctx, FT_ERR_WAIT_TMEM_EMPTY)) {
              ok = false;
              continue;
            }
            if ((seen >> t) & 1u) blk ^= 1u << t;
            seen |= 1u << t;
            tc_fence_after();
            if (elect_one()) {
              mma_kmajor<HD>(tmem_base + C::TM_S + 128 * t, q_addr + q_slot[t] * C::TILE, k_addr + rk.s * C::TILE, idesc_s);
              umma_commit(&s_full[t]);
            }
            __syncwarp();
          }
          if (!ok) break;
          if (elect_one()) umma_commit(&k_empty[rk.s]);
          __syncwarp();
          rk.step();
        }
      }
    } else if (warp == 10) {
      // ------------------------------------------------------------ MMA issuer 2: O += P V
      const uint32_t idesc_pv = make_idesc_bf16(128, HD, 0, 1);
      const uint32_t v_addr = smem_u32(smem + C::OFF_V);
      Ring<C::VS> rv;
      uint32_t blk = 0, used = 0, freed = 0;   // bit t: parity of the tile's block; an earlier item used it; parity of o_free
      bool ok = true;
#pragma unroll 1
      for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
        const FwdItem it(item, p);
#pragma unroll 1
        for (int j = 0; ok && j < it.nkv; ++j) {
          if (!mbar_wait_warp(&v_full[rv.s], rv.ph, ctx, FT_ERR_WAIT_FULL)) { ok = false; break; }
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!ok || j >= it.nb[t]) continue;
            const uint32_t par = (blk >> t) & 1u;
            if (!mbar_wait_warp(&p_ready[t], par, ctx, FT_ERR_WAIT_SOFTMAX)) { ok = false; continue; }
            blk ^= 1u << t;
            if (j == 0) {
              // the accumulator still holds the previous item's output until its group has read it
              if (((used >> t) & 1u) && !mbar_wait_warp(&o_free[t], (freed >> t) & 1u, ctx, FT_ERR_WAIT_TMEM_EMPTY)) {
                ok = false;
                continue;
              }
              if ((used >> t) & 1u) freed ^= 1u << t;
              used |= 1u << t;
            }
            // the first 64 keys are multiplied under the exponentials of the other 64
            const uint32_t o_tmem = tmem_base + C::TM_O + HD * t, p_tmem = tmem_base + C::TM_P + C::P_STRIDE * t;
            tc_fence_after();
            if (elect_one()) mma_ptmem_times_rows<0, 4>(o_tmem, p_tmem, v_addr + rv.s * C::TILE, idesc_pv, j > 0);
            __syncwarp();
            if (!mbar_wait_warp(&p_ready[2 + t], par, ctx, FT_ERR_WAIT_SOFTMAX)) { ok = false; continue; }
            tc_fence_after();
            if (elect_one()) {
              mma_ptmem_times_rows<4, 8>(o_tmem, p_tmem, v_addr + rv.s * C::TILE, idesc_pv, true);
              umma_commit(&pv_done[t]);
            }
            __syncwarp();
          }
          if (!ok) break;
          if (elect_one()) umma_commit(&v_empty[rv.s]);
          __syncwarp();
          rv.step();
        }
      }
    }
  } else {
    // ------------------------------------------------------------ softmax groups
    reg_inc<216>();
    const int t = warp >> 2;                 // tile of this group
    const int qd = warp & 3;
    const int row = qd * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(qd * 32) << 16;
    const uint32_t s_tmem = tmem_base + C::TM_S + 128 * t + lane_sel;
    const uint32_t o_tmem = tmem_base + C::TM_O + HD * t + lane_sel;
    const uint32_t p_tmem = tmem_base + C::TM_P + C::P_STRIDE * t + lane_sel;
    const f32x2 sl2 = pk2(p.sl2, p.sl2);
    uint32_t blk = 0;                        // parity of the tile's block
    Ring<C::QS> rq;                          // the Q tile of the group's next item
    AttnTurns turns;
    bool ok = true;
#pragma unroll 1
    for (int item = walk.next(); ok && item >= 0; item = walk.next()) {
      const FwdItem it(item, p);
      const int n_my = t == 0 ? it.nb[0] : it.nb[1], n_other = t == 0 ? it.nb[1] : it.nb[0];
      turns.item(n_my, n_other);
      if (t == 1 && n_other > 0) rq.step();         // tile 0's Q comes first
      const int q_slot = rq.s;
      if (n_my > 0) rq.step();
      if (t == 0 && n_other > 0) rq.step();
      if (n_my == 0) continue;
      const int grow = it.q0 + t * AT_T + row;
      const int last_col = p.causal ? min(grow, p.S - 1) : p.S - 1;                            // last valid key of this row
      const int warp_last = p.causal ? min(it.q0 + t * AT_T + qd * 32, p.S - 1) : p.S - 1;    // of the warp's first row
      float m2 = -INFINITY;                    // reference maximum, already times sl2
      float l = 0.f;
#pragma unroll 1
      for (int j = 0; j < n_my; ++j) {
        if (!mbar_wait_warp(&s_full[t], blk, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
        uint32_t r[128];
        tmem_ld32(s_tmem + 0, r + 0);
        tmem_ld32(s_tmem + 32, r + 32);
        tmem_ld32(s_tmem + 64, r + 64);
        tmem_ld32(s_tmem + 96, r + 96);
        tmem_ld_wait();
        if constexpr (!C::ALIAS) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_free[t]);   // the next QK^T may overwrite the score tile now
        }
        const int k0 = j * AT_T;
        if (k0 + AT_T - 1 > warp_last) {
          const int lim = last_col - k0;
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i > lim) r[i] = __float_as_uint(-INFINITY);
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 128; i += 8) {
          mx0 = max3(mx0, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
          mx1 = max3(mx1, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
          mx2 = max3(mx2, __uint_as_float(r[i + 4]), __uint_as_float(r[i + 5]));
          mx3 = max3(mx3, __uint_as_float(r[i + 6]), __uint_as_float(r[i + 7]));
        }
        const float bm2 = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * p.sl2;   // sl2 > 0
        // lazy reference maximum: move it only when this block exceeds the headroom
        float alpha = 1.f;
        const bool move = (bm2 > m2 + F2_LAZY) || (m2 == -INFINITY && bm2 > -INFINITY);
        if (move) {
          alpha = (m2 == -INFINITY) ? 0.f : fast_exp2(m2 - bm2);
          m2 = bm2;
        }
        const float moff = (m2 == -INFINITY) ? 0.f : -m2;
        const f32x2 off = pk2(moff, moff);
        f32x2 rs0 = pk2(0.f, 0.f), rs1 = rs0;
        // exponentials of elements [i0, i0 + 64): packed probabilities reuse the low registers
        auto exp_half = [&](int i0) {
#pragma unroll
          for (int i = i0; i < i0 + 64; i += 4) {
            const f32x2 e0 = exp2_pair(fma2(acc2(r, i), sl2, off));
            const f32x2 e1 = exp2_pair(fma2(acc2(r, i + 2), sl2, off));
            rs0 = add2(rs0, e0);
            rs1 = add2(rs1, e1);
            r[i >> 1] = pack2(e0);
            r[(i >> 1) + 1] = pack2(e1);
          }
        };
        // PV of the previous block must be finished before P is overwritten and before the
        // accumulator may be rescaled
        if (j > 0) {
          if (!mbar_wait_warp(&pv_done[t], blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
          tc_fence_after();
          if (__any_sync(0xffffffffu, move)) {
#pragma unroll
            for (int c = 0; c < HD; c += 32) {
              uint32_t v[32];
              tmem_ld32(o_tmem + c, v);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
              tmem_st32(o_tmem + c, v);
            }
          }
        }
        // The groups take turns (see AttnTurns).  Side by side they halve each other's rate on the one unit that evaluates
        // exponentials, and both groups' other work then leaves it idle (1 x 1500 x 20 heads of 64: 26.0 us side by side,
        // 23.5 us in turns).  With head_dim 128 the score products keep the groups apart by themselves (4 x 2048 x 16, causal:
        // 77.5 us in turns, 75.3 us without).  Every wait is for work that precedes this block in the order (item, block,
        // tile) in which scores, products and turns are issued, so the turns add no cycle to the other barriers.
        uint32_t turn;
        if (C::TURNS && turns.waits(t, j, turn)) {
          if (!mbar_wait_warp(&e_done[t ^ 1], turn, ctx, FT_ERR_WAIT_WARPS)) { ok = false; break; }
        }
        // probabilities go to tensor memory, each half as soon as it is computed
        exp_half(0);
        tmem_st32(p_tmem, r);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[t]);
        exp_half(64);
        if (C::TURNS && turns.takes(j) && lane == 0) mbar_arrive(&e_done[t]);
        tmem_st32(p_tmem + 32, r + 32);
        const float2 s0 = up2(add2(rs0, rs1));
        l = l * alpha + (s0.x + s0.y);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[2 + t]);
        blk ^= 1u;
      }
      if (!ok || !mbar_wait_warp(&pv_done[t], blk ^ 1u, ctx, FT_ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint32_t v[HD];
#pragma unroll
      for (int c = 0; c < HD; c += 32) tmem_ld32(o_tmem + c, v + c);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_free[t]);
      // The output leaves through the warp's 32 rows of the Q tile, which the scores no longer need, by the TMA unit, which cuts
      // off the rows past the end.  (Read back and stored 128 bytes of a row by eight lanes: B8 S1024 H12 head size 64 causal 27.6 us,
      // 26.6 so; 1 x 1500 x 20 21.8 and 21.6; head size 128 unchanged.  Leaving it behind the next item's first block, as the
      // backward kernels do, cost the block loop registers: 30.3 -> 32.1 us.)
      const int r0 = it.q0 + t * AT_T + qd * 32;
      uint8_t* stage = smem + C::OFF_Q + q_slot * C::TILE + qd * 32 * 128;
#pragma unroll
      for (int c = 0; c < HD; c += 64) {
#pragma unroll
        for (int i = 0; i < 64; i += 8) {
          uint4 u;
          u.x = pack_bf16(__uint_as_float(v[c + i + 0]) * inv, __uint_as_float(v[c + i + 1]) * inv);
          u.y = pack_bf16(__uint_as_float(v[c + i + 2]) * inv, __uint_as_float(v[c + i + 3]) * inv);
          u.z = pack_bf16(__uint_as_float(v[c + i + 4]) * inv, __uint_as_float(v[c + i + 5]) * inv);
          u.w = pack_bf16(__uint_as_float(v[c + i + 6]) * inv, __uint_as_float(v[c + i + 7]) * inv);
          *reinterpret_cast<uint4*>(stage + (c / 64) * AT_REGION + lane * 128 + (((i >> 3) ^ (lane & 7)) << 4)) = u;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (r0 < p.S) {
#pragma unroll
          for (int c = 0; c < HD; c += 64) tma_store_4d(&tmO, stage + (c / 64) * AT_REGION, c, r0, it.h, it.b);
          bulk_wait_read_all();
        }
        mbar_arrive(&q_empty[q_slot]);       // the tile goes back to the loader
      }
      if (p.lse && grow < p.S)
        p.lse[((long long)it.b * p.H + it.h) * p.S + grow] = (l > 0.f) ? m2 + log2f(l) : -INFINITY;
    }
  }

  if (*abort_f) {
    for (int i = 0; i < 100; ++i) __nanosleep(10000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

template <int HD>
static int attn_fwd2_launch(const FtkAttnDesc* a, cudaStream_t s) {
  CUtensorMap tq, tk, tv, to;
  int rc;
  if ((rc = make_map(&tq, a->q, a, a->q_bs, a->q_ss, a->q_hs))) return rc;
  if ((rc = make_map(&tk, a->k, a, a->k_bs, a->k_ss, a->k_hs))) return rc;
  if ((rc = make_map(&tv, a->v, a, a->v_bs, a->v_ss, a->v_hs))) return rc;
  // (the stride of an extent of one is never stepped over and may be anything)
  if ((rc = make_map(&to, a->o, a, a->B > 1 ? a->o_bs : 0, a->S > 1 ? a->o_ss : a->hd, a->H > 1 ? a->o_hs : 0, 64, 32))) return rc;
  AttnArgs p{};
  fill_args(p, a);
  if (!p.status) return -6;
  static bool attr = false;
  if (!attr) {
    if ((rc = set_smem(attn_fwd2_kernel<HD>, Fwd2Cfg<HD>::SMEM))) return rc;
    attr = true;
  }
  unsigned grid = 0;
  if ((rc = set_items(p, a, 2 * AT_T, &grid))) return rc;
  launch_pdl(attn_fwd2_kernel<HD>, grid, F2_THREADS, Fwd2Cfg<HD>::SMEM, s, tq, tk, tv, to, p);
  return (int)cudaGetLastError();
}

}  // namespace ftk

using namespace ftk;

extern "C" int ftk_attn_fwd(const FtkAttnDesc* a, void* stream) {
  if (!a || a->B <= 0 || a->H <= 0 || a->S <= 0) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a->hd == 64) return attn_fwd2_launch<64>(a, s);
  if (a->hd == 128) return attn_fwd2_launch<128>(a, s);
  return -5;
}
