// Row-wise kernels: LayerNorm / RMSNorm forward+backward, softmax, fused
// softmax-cross-entropy, fixed-tree reductions.  All memory bound: one pass over
// the data where it fits on chip, 16-byte vector accesses, fp32 statistics.
//
// Semantics follow the reference CPU kernels: two-pass LayerNorm with population
// variance (ft-kernel-cpu/src/lib.rs:5824), RMSNorm (:6418, backward :6503),
// cross-entropy = lse - logit[target] with gradient softmax - onehot (:6649,:6679),
// guarded row softmax of the Metal shader (ft-kernel-metal/src/fused.rs:321).
// Parameter-gradient reductions run in a fixed order (row blocks, then a fixed tree over
// the block partials), so two runs give identical bits.
#include "ft_sm100.cuh"
#include "launch.cuh"
#include "ftk_api.h"

namespace ftk {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]);
  u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  return u;
}

// The same as pairs, two values per instruction from here on.
__device__ __forceinline__ void unpack4x2(const uint4& u, f32x2* f) {
  f[0] = unpack_bf16_2(u.x); f[1] = unpack_bf16_2(u.y); f[2] = unpack_bf16_2(u.z); f[3] = unpack_bf16_2(u.w);
}
__device__ __forceinline__ uint32_t pack_pair(f32x2 a) {
  const float2 f = up2(a);
  return pack_bf16(f.x, f.y);
}
__device__ __forceinline__ uint4 pack4x2(const f32x2* f) {
  return make_uint4(pack_pair(f[0]), pack_pair(f[1]), pack_pair(f[2]), pack_pair(f[3]));
}
__device__ __forceinline__ float hsum(f32x2 a) {
  const float2 f = up2(a);
  return f.x + f.y;
}

constexpr int ROW_WARPS = 8;     // rows per CTA

// ----------------------------------------------------------------------------- LayerNorm fwd
// Rows of up to 256 NV columns: a warp owns a row and keeps it in registers, NV 16-byte vectors per lane; wider rows (up to
// 16384 columns) are shared by the four or eight warps of a CTA.  The row, gamma and beta are all requested before the first
// addition, so a row costs one memory latency; a warp that re-reads columns beyond its registers, as it did from 1024
// columns on, pays three.  Sums run over a lane's vectors in ascending order, then over the lanes (and warps) in a fixed tree.
// Memory bound (captured loop, L2 warm): 8192 x 768 6.9 -> 5.3 us (25 MB), 8192 x 2048 14.6 -> 11.6, 1500 x 1280 5.6 -> 3.3; pairs of values per
// instruction (f32x2) are a third of the first: the kernel was at two thirds of its issue slots.
// LEAN: gamma and beta are read at the end, which leaves registers for 32 warps per SM instead of 20.  Only four vectors per
// lane and many rows gain: 65536 x 1024 51.4 -> 43.4 us (RMS 46.7 -> 40.7), 4096 x 1024 4.6 -> 3.9, but 500 x 1024 2.2 -> 2.8.
// (No bound, 0, for the others: a bound of one block lets the compiler take 130 registers for six vectors, and 8192 x 1536
// goes from 9.5 to 10.5 us.)
template <int NV, int WPR, bool RMS, bool LEAN = false>
__global__ void __launch_bounds__(WPR == 8 ? 256 : 128, LEAN ? 8 : 0)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ resid,
                __nv_bfloat16* __restrict__ sum_out, const __nv_bfloat16* __restrict__ gamma,
                const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int cols,
                float eps) {
  pdl_wait();
  if constexpr (WPR == 1)
    pdl_trigger_work(4 * cols * 4);
  else
    pdl_trigger();       // 6 KB and more (and RMSNorm of two vectors a lane keeps its 48 registers)
  __shared__ float red[2][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = WPR == 1 ? blockIdx.x * 4 + warp : blockIdx.x;
  const int v0 = WPR == 1 ? lane : (int)threadIdx.x;
  constexpr int STEP = 32 * WPR;
  if (row >= rows) return;
  const int nvec = cols >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * cols);
  const uint4* rr = resid ? reinterpret_cast<const uint4*>(resid + (size_t)row * cols) : nullptr;
  const uint4* gv = reinterpret_cast<const uint4*>(gamma);
  const uint4* bv = reinterpret_cast<const uint4*>(beta);
  constexpr bool PRE = NV <= 6 && !LEAN;      // more vectors than that: gamma and beta come from L1 at the end, for the registers' sake
  uint4 xc[NV], rc[NV], gc[PRE ? NV : 1], bc[PRE ? NV : 1];
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const int v = v0 + STEP * c;
    xc[c] = rc[c] = make_uint4(0u, 0u, 0u, 0u);
    if (v < nvec) {
      xc[c] = xr[v];
      if (rr) rc[c] = rr[v];
    }
  }
  auto affine = [&](int c, uint4& g, uint4& b) {
    const int v = v0 + STEP * c;
    g = b = make_uint4(0u, 0u, 0u, 0u);
    if (v < nvec) {
      g = __ldg(gv + v);
      if (beta) b = __ldg(bv + v);
    }
  };
  if (PRE) {
#pragma unroll
    for (int c = 0; c < NV; ++c) affine(c, gc[PRE ? c : 0], bc[PRE ? c : 0]);
  }
  auto row_sum = [&](float v, int slot) -> float {
    v = warp_sum(v);
    if (WPR > 1) {
      if (lane == 0) red[slot][warp] = v;
      __syncthreads();
      v = red[slot][0];
#pragma unroll
      for (int w = 1; w < WPR; ++w) v += red[slot][w];
    }
    return v;
  };
  f32x2 f[NV][4];
  f32x2 s2 = pk2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    unpack4x2(xc[c], f[c]);
    if (rr) {
      f32x2 g[4];
      unpack4x2(rc[c], g);
#pragma unroll
      for (int i = 0; i < 4; ++i) f[c][i] = add2(f[c][i], g[i]);
      const uint4 u = pack4x2(f[c]);
      unpack4x2(u, f[c]);  // statistics are taken on the rounded sum that downstream kernels will read
      if (sum_out && v0 + STEP * c < nvec) reinterpret_cast<uint4*>(sum_out + (size_t)row * cols)[v0 + STEP * c] = u;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) s2 = RMS ? fma2(f[c][i], f[c][i], s2) : add2(s2, f[c][i]);
  }
  const float s = row_sum(hsum(s2), 0);
  float mean = 0.f, rstd;
  if (RMS) {
    rstd = rsqrtf(s / cols + eps);
  } else {
    mean = s / cols;
    const f32x2 nm = pk2(-mean, -mean);
    f32x2 q2 = pk2(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < NV; ++c)
      if (v0 + STEP * c < nvec) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          f[c][i] = add2(f[c][i], nm);
          q2 = fma2(f[c][i], f[c][i], q2);
        }
      }
    rstd = rsqrtf(row_sum(hsum(q2), 1) / cols + eps);
  }
  if (v0 == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
  const f32x2 rs = pk2(rstd, rstd);
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * cols);
#pragma unroll
  for (int c = 0; c < NV; ++c)
    if (v0 + STEP * c < nvec) {
      f32x2 g[4], b[4];
      if (!PRE) affine(c, gc[0], bc[0]);
      unpack4x2(gc[PRE ? c : 0], g);
      unpack4x2(bc[PRE ? c : 0], b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const f32x2 h = mul2(f[c][i], rs);
        f[c][i] = beta ? fma2(h, g[i], b[i]) : mul2(h, g[i]);
      }
      yr[v0 + STEP * c] = pack4x2(f[c]);
    }
}

// Rows of more than 16384 columns: the eight warps of a CTA walk the row three times.
template <bool RMS>
__global__ void __launch_bounds__(ROW_WARPS * 32)
norm_fwd_long_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ resid,
                     __nv_bfloat16* __restrict__ sum_out, const __nv_bfloat16* __restrict__ gamma,
                     const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int cols,
                     float eps) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[2][ROW_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x;
  auto row_sum = [&](float v, int slot) -> float {
    v = warp_sum(v);
    if (lane == 0) red[slot][warp] = v;
    __syncthreads();
    v = red[slot][0];
#pragma unroll
    for (int w = 1; w < ROW_WARPS; ++w) v += red[slot][w];
    return v;
  };
  const int nvec = cols >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * cols);
  const uint4* rr = resid ? reinterpret_cast<const uint4*>(resid + (size_t)row * cols) : nullptr;
  uint4* so = sum_out ? reinterpret_cast<uint4*>(sum_out + (size_t)row * cols) : nullptr;
  const uint4* src = rr ? reinterpret_cast<const uint4*>(so) : xr;
  float s = 0.f;
  for (int v = threadIdx.x; v < nvec; v += ROW_WARPS * 32) {
    float f[8];
    unpack8(xr[v], f);
    if (rr) {
      float g[8];
      unpack8(rr[v], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
      const uint4 u = pack8(f);
      unpack8(u, f);
      if (so) so[v] = u;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) s += RMS ? f[i] * f[i] : f[i];
  }
  s = row_sum(s, 0);
  float mean = 0.f, rstd;
  if (RMS) {
    rstd = rsqrtf(s / cols + eps);
  } else {
    mean = s / cols;
    float q = 0.f;
    for (int v = threadIdx.x; v < nvec; v += ROW_WARPS * 32) {
      float f[8];
      unpack8(src[v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d = f[i] - mean;
        q += d * d;
      }
    }
    q = row_sum(q, 1);
    rstd = rsqrtf(q / cols + eps);
  }
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
  const uint4* gv = reinterpret_cast<const uint4*>(gamma);
  const uint4* bv = beta ? reinterpret_cast<const uint4*>(beta) : nullptr;
  uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * cols);
  for (int v = threadIdx.x; v < nvec; v += ROW_WARPS * 32) {
    float f[8], g[8], b[8];
    unpack8(src[v], f);
    unpack8(__ldg(gv + v), g);
    if (bv) unpack8(__ldg(bv + v), b);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float h = (f[i] - mean) * rstd * g[i];
      f[i] = bv ? h + b[i] : h;
    }
    yr[v] = pack8(f);
  }
}

// ----------------------------------------------------------------------------- LayerNorm bwd dx
template <bool RMS>
__global__ void __launch_bounds__(ROW_WARPS * 32)
norm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean_in,
                   const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dx_add,
                   __nv_bfloat16* __restrict__ dx, int rows, int cols) {
  pdl_wait();
  pdl_trigger_work(ROW_WARPS * cols * 6);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * ROW_WARPS + warp;
  if (row >= rows) return;
  const int nvec = cols >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * cols);
  const uint4* dr = reinterpret_cast<const uint4*>(dy + (size_t)row * cols);
  const uint4* gv = reinterpret_cast<const uint4*>(gamma);
  const float mean = RMS ? 0.f : mean_in[row];
  const float rstd = rstd_in[row];
  // sums of g*dy and g*dy*xhat
  float s1 = 0.f, s2 = 0.f;
  for (int v = lane; v < nvec; v += 32) {
    float fx[8], fd[8], g[8];
    unpack8(xr[v], fx);
    unpack8(dr[v], fd);
    unpack8(__ldg(gv + v), g);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float gd = g[i] * fd[i];
      float xh = (fx[i] - mean) * rstd;
      s1 += gd;
      s2 += gd * xh;
    }
  }
  s1 = warp_sum(s1) / cols;
  s2 = warp_sum(s2) / cols;
  if (RMS) s1 = 0.f;
  const uint4* av = dx_add ? reinterpret_cast<const uint4*>(dx_add + (size_t)row * cols) : nullptr;
  uint4* ov = reinterpret_cast<uint4*>(dx + (size_t)row * cols);
  for (int v = lane; v < nvec; v += 32) {
    float fx[8], fd[8], g[8], a[8];
    unpack8(xr[v], fx);
    unpack8(dr[v], fd);
    unpack8(__ldg(gv + v), g);
    if (av) unpack8(av[v], a);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float xh = (fx[i] - mean) * rstd;
      float r = rstd * (g[i] * fd[i] - s1 - xh * s2);
      fx[i] = av ? r + a[i] : r;
    }
    ov[v] = pack8(fx);
  }
}

// ----------------------------------------------------------------------------- norm bwd, one pass
// dx and the per-block column partials of dgamma / dbeta from a single read of dy and x (and of the gradient that is added to
// dx), rows of up to 8192 columns.  A CTA of 8 warps owns a contiguous range of rows and takes them in steps of G = 8 / WPR
// rows, WPR warps per row, NV 16-byte vectors per lane.  The rows of a step are one contiguous piece of each array: bulk
// copies bring it into a ring of shared-memory stages, so the bytes in flight per SM do not depend on registers.  Column
// sums of dy * xhat and dy stay in registers; at the end the G groups' sums are added in group order and the CTA writes
// partial[blk][c].  Rows go to CTAs and warps by index alone, so the result does not depend on scheduling.
// Memory bound from some thousand rows on: with the gradient that is added, column sums finished, 8192 x 768 17.9 -> 15.9 us
// (one row per warp prefetched in registers before), 8192 x 2048 62.9 -> 37.1 us and 1500 x 1280 15.8 -> 10.6 us (three
// kernels before: rows wider than 768 columns spilled the column sums of one warp per row).
constexpr int NB_MAX_BLOCKS = 296;       // two CTAs per SM
constexpr int NB_RING_BYTES = 96 * 1024; // operand stages of one CTA
template <int NV, int WPR, bool RMS>
__global__ void __launch_bounds__(ROW_WARPS * 32, 2)
norm_bwd_fused_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                      const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean_in,
                      const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dx_add,
                      __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int rows, int cols,
                      int rows_per_blk, int stages, int* status) {
  constexpr int G = ROW_WARPS / WPR;
  extern __shared__ __align__(128) uint8_t nb_smem[];
  __shared__ uint64_t full[8], empty[8];
  __shared__ int abort_w;
  __shared__ float red[2][ROW_WARPS][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = warp / WPR;                            // row of the step
  const int v0 = (warp % WPR) * 32 + lane;               // first vector of this lane
  constexpr int STEP = 32 * WPR;
  const int nvec = cols >> 3;
  const int n_arr = dx_add ? 3 : 2;
  const uint32_t piece = (uint32_t)(G * cols * 2);       // bytes of one array in one stage
  WaitCtx ctx{status, &abort_w};
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], ROW_WARPS);
    }
    abort_w = 0;
    fence_mbar_init();
  }
  pdl_wait();
  pdl_trigger();
  uint4 gam[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j)
    gam[j] = v0 + STEP * j < nvec ? __ldg(reinterpret_cast<const uint4*>(gamma) + v0 + STEP * j) : make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const int row_begin = blockIdx.x * rows_per_blk, row_end = min(rows, row_begin + rows_per_blk);
  const int steps = row_end > row_begin ? (row_end - row_begin + G - 1) / G : 0;
  auto load_step = [&](int st) {       // one thread
    const int r = row_begin + st * G, n = min(G, row_end - r);
    uint8_t* dst = nb_smem + (size_t)(st % stages) * n_arr * piece;
    uint64_t* bar = &full[st % stages];
    const uint32_t bytes = (uint32_t)(n * cols * 2);
    mbar_arrive_expect_tx(bar, n_arr * bytes);
    auto copy = [&](int a, const __nv_bfloat16* src) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(smem_u32(dst + a * piece)), "l"(src + (size_t)r * cols), "r"(bytes), "r"(smem_u32(bar))
                   : "memory");
    };
    copy(0, x);
    copy(1, dy);
    if (dx_add) copy(2, dx_add);
  };
  if ((int)threadIdx.x < stages && (int)threadIdx.x < steps) load_step((int)threadIdx.x);      // one thread per stage
  f32x2 dg[NV][4], db[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) dg[j][i] = db[j][i] = pk2(0.f, 0.f);
  bool ok = true;
  float mean_n = 0.f, rstd_n = 0.f;
  auto fetch_stats = [&](int st) {
    const int row = row_begin + st * G + grp;
    if (row < row_end) {
      mean_n = RMS ? 0.f : __ldg(mean_in + row);
      rstd_n = __ldg(rstd_in + row);
    }
  };
  fetch_stats(0);
  for (int st = 0; st < steps; ++st) {
    const int row = row_begin + st * G + grp;
    const bool live = row < row_end;
    const float mean = mean_n, rstd = rstd_n;
    fetch_stats(st + 1);
    if (ok) ok = mbar_wait(&full[st % stages], (st / stages) & 1, ctx, FT_ERR_WAIT_FULL);
    const uint8_t* src = nb_smem + (size_t)(st % stages) * n_arr * piece + (size_t)grp * cols * 2;
    const uint4* xv = reinterpret_cast<const uint4*>(src);
    const uint4* dv = reinterpret_cast<const uint4*>(src + piece);
    const uint4* av = reinterpret_cast<const uint4*>(src + 2 * piece);
    const f32x2 nm = pk2(-mean, -mean), rs = pk2(rstd, rstd);
    f32x2 a1 = pk2(0.f, 0.f), a2 = a1;
    if (live && ok) {
#pragma unroll
      for (int j = 0; j < NV; ++j)
        if (v0 + STEP * j < nvec) {
          f32x2 fx[4], fd[4], g[4];
          unpack4x2(xv[v0 + STEP * j], fx);
          unpack4x2(dv[v0 + STEP * j], fd);
          unpack4x2(gam[j], g);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const f32x2 gd = mul2(g[i], fd[i]);
            const f32x2 xh = mul2(RMS ? fx[i] : add2(fx[i], nm), rs);
            if (!RMS) a1 = add2(a1, gd);
            a2 = fma2(gd, xh, a2);
            dg[j][i] = fma2(fd[i], xh, dg[j][i]);
            if (!RMS) db[j][i] = add2(db[j][i], fd[i]);
          }
        }
    }
    float s1 = RMS ? 0.f : hsum(a1), s2 = hsum(a2);
    if (!RMS) s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (WPR > 1) {
      if (lane == 0) {
        red[st & 1][warp][0] = s1;
        red[st & 1][warp][1] = s2;
      }
      __syncthreads();
      s1 = s2 = 0.f;
#pragma unroll
      for (int w = 0; w < WPR; ++w) {
        s1 += red[st & 1][grp * WPR + w][0];
        s2 += red[st & 1][grp * WPR + w][1];
      }
    }
    const f32x2 m1 = pk2(-s1 / cols, -s1 / cols), m2 = pk2(-s2 / cols, -s2 / cols);
    if (live && ok) {
      uint4* ov = reinterpret_cast<uint4*>(dx + (size_t)row * cols);
#pragma unroll
      for (int j = 0; j < NV; ++j)
        if (v0 + STEP * j < nvec) {
          f32x2 fx[4], fd[4], g[4], a[4];
          unpack4x2(xv[v0 + STEP * j], fx);
          unpack4x2(dv[v0 + STEP * j], fd);
          unpack4x2(gam[j], g);
          if (dx_add) unpack4x2(av[v0 + STEP * j], a);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const f32x2 xh = mul2(RMS ? fx[i] : add2(fx[i], nm), rs);
            f32x2 t = mul2(g[i], fd[i]);
            if (!RMS) t = add2(t, m1);
            t = fma2(xh, m2, t);
            fx[i] = dx_add ? fma2(rs, t, a[i]) : mul2(rs, t);
          }
          ov[v0 + STEP * j] = pack4x2(fx);
        }
    }
    fence_proxy_async_smem();            // this warp has read its part of the stage
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st % stages]);
    // the stage of the step before (the other warps have left it by now) takes the next rows
    if (threadIdx.x == 0 && ok && st > 0 && st - 1 + stages < steps) {
      if (mbar_wait(&empty[(st - 1) % stages], ((st - 1) / stages) & 1, ctx, FT_ERR_WAIT_EMPTY)) load_step(st - 1 + stages);
    }
  }
  // the groups' column sums, added in group order: dgamma first, then dbeta
  if (!partial) return;
  constexpr int NS = RMS ? 1 : 2;                        // dgamma, dbeta
  float* acc = reinterpret_cast<float*>(nb_smem);        // [NS][G][cols], in the stages
  __syncthreads();                                       // the stages have been read
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    float* d0 = G > 1 ? acc + (size_t)(k * G + grp) * cols : partial + ((size_t)k * gridDim.x + blockIdx.x) * cols;
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (v0 + STEP * j < nvec) {
        float* d = d0 + (v0 + STEP * j) * 8;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 lo = up2(k ? db[j][2 * h] : dg[j][2 * h]), hi = up2(k ? db[j][2 * h + 1] : dg[j][2 * h + 1]);
          reinterpret_cast<float4*>(d)[h] = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
      }
  }
  if (G == 1) return;
  __syncthreads();
  for (int c = threadIdx.x * 4; c < cols; c += blockDim.x * 4) {
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      float4 t = *reinterpret_cast<const float4*>(acc + (size_t)k * G * cols + c);
#pragma unroll
      for (int g = 1; g < G; ++g) {
        const float4 u = *reinterpret_cast<const float4*>(acc + (size_t)(k * G + g) * cols + c);
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
      *reinterpret_cast<float4*>(partial + ((size_t)k * gridDim.x + blockIdx.x) * cols + c) = t;
    }
  }
}

// Fixed-order sum over block partials.  G groups share a column: group g adds partial[b][c] for b = g, g + G, ... ascending with
// up to eight loads of each array in flight, then the group sums are added, in group order (G = 8) or by a fixed shuffle tree
// (G = 32).  A second array (dbeta) goes along.  All latency, so the number of groups follows the number of partials, see
// col_final().
template <int G>
__global__ void __launch_bounds__(G == 1 ? 128 : 32 * G)
col_final_kernel(const float* __restrict__ partial, float* __restrict__ out,
                 const float* __restrict__ partial2, float* __restrict__ out2, int cols, int nblk,
                 int accumulate) {
  pdl_wait();
  pdl_trigger();
  constexpr int CW = G == 1 ? 128 : 32;                  // columns of a CTA
  __shared__ float sm[2][G][CW + 1];
  const int cl = threadIdx.x % CW, g = threadIdx.x / CW;
  const int c = blockIdx.x * CW + cl;
  float s = 0.f, t = 0.f;
  if (c < cols) {
    for (int b0 = g; b0 < nblk; b0 += G * 8) {
      float u[8], w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int b = b0 + G * k;
        u[k] = b < nblk ? partial[(size_t)b * cols + c] : 0.f;
        w[k] = (partial2 && b < nblk) ? partial2[(size_t)b * cols + c] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s += u[k];
        t += w[k];
      }
    }
  }
  if constexpr (G > 1) {
    sm[0][g][cl] = s;
    sm[1][g][cl] = t;
    __syncthreads();
    if constexpr (G == 32) {
      // warp g now owns column g of the 32; lane = group
      s = warp_sum(sm[0][cl][g]);
      t = partial2 ? warp_sum(sm[1][cl][g]) : 0.f;
    } else if (g == 0) {
      s = t = 0.f;
#pragma unroll
      for (int k = 0; k < G; ++k) {
        s += sm[0][k][cl];
        t += sm[1][k][cl];
      }
    }
  }
  const int cc = G == 32 ? blockIdx.x * 32 + g : c;
  if ((G == 32 ? cl : g) == 0 && cc < cols) {
    out[cc] = accumulate ? out[cc] + s : s;
    if (partial2) out2[cc] = accumulate ? out2[cc] + t : t;
  }
}

// Column partials: partial[blk][c] = sum over this block's rows of dy*xhat, and of dy.
// MODE 0: LayerNorm (two outputs), 1: RMSNorm (dgamma only), 2: plain column sum of dy.
// A CTA covers 64 columns x COL_ROWS_PER_BLK rows with 8 row groups of 32 column pairs:
// each thread sums its rows in ascending order, then thread (group 0) adds the 8 group
// sums in ascending group order - a fixed tree, independent of scheduling.
constexpr int COL_ROWS_PER_BLK = 256;
constexpr int COL_GROUPS = 8;
template <int MODE>
__global__ void __launch_bounds__(256)
col_partial_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                   float* __restrict__ partial, int rows, int cols, long long ld, int nblk) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sm[4][COL_GROUPS][32];
  const int cp = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + cp) * 2;
  const int blk = blockIdx.y;
  const int r0 = blk * COL_ROWS_PER_BLK;
  const int r1 = min(rows, r0 + COL_ROWS_PER_BLK);
  float g0 = 0.f, g1 = 0.f, b0 = 0.f, b1 = 0.f;
  if (c < cols) {
    for (int r = r0 + rg; r < r1; r += COL_GROUPS) {
      float2 d = unpack_bf16(*reinterpret_cast<const uint32_t*>(dy + (size_t)r * ld + c));
      if (MODE == 2) {
        b0 += d.x; b1 += d.y;
      } else {
        float2 xv = unpack_bf16(*reinterpret_cast<const uint32_t*>(x + (size_t)r * ld + c));
        float mu = MODE == 0 ? mean_in[r] : 0.f;
        float rs = rstd_in[r];
        g0 += d.x * (xv.x - mu) * rs;
        g1 += d.y * (xv.y - mu) * rs;
        b0 += d.x; b1 += d.y;
      }
    }
  }
  sm[0][rg][cp] = g0; sm[1][rg][cp] = g1; sm[2][rg][cp] = b0; sm[3][rg][cp] = b1;
  __syncthreads();
  if (rg == 0 && c < cols) {
    float t0 = 0.f, t1 = 0.f, t2 = 0.f, t3 = 0.f;
#pragma unroll
    for (int k = 0; k < COL_GROUPS; ++k) {
      t0 += sm[0][k][cp]; t1 += sm[1][k][cp]; t2 += sm[2][k][cp]; t3 += sm[3][k][cp];
    }
    if (MODE == 2) {
      partial[(size_t)blk * cols + c] = t2;
      if (c + 1 < cols) partial[(size_t)blk * cols + c + 1] = t3;
    } else {
      partial[(size_t)blk * cols + c] = t0;
      if (c + 1 < cols) partial[(size_t)blk * cols + c + 1] = t1;
      if (MODE == 0) {
        float* pb = partial + (size_t)nblk * cols;
        pb[(size_t)blk * cols + c] = t2;
        if (c + 1 < cols) pb[(size_t)blk * cols + c + 1] = t3;
      }
    }
  }
}
// ----------------------------------------------------------------------------- softmax
template <typename T>
__device__ __forceinline__ float ldf(const T* p);
template <>
__device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <typename T>
__device__ __forceinline__ void stf(T* p, float v);
template <>
__device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <>
__device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16(v);
}

__device__ __forceinline__ float block_reduce(float v, float* red, bool is_max) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : (is_max ? -INFINITY : 0.f);
    t = is_max ? warp_max(t) : warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// One CTA per row; `limit` = number of valid columns in this row (causal rows pass row+1).
template <typename T>
__global__ void __launch_bounds__(256)
softmax_rows_kernel(const T* __restrict__ x, T* __restrict__ y, int cols, int S_causal,
                    float scale) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const int limit = S_causal > 0 ? (int)(row % S_causal) + 1 : cols;
  const T* xr = x + row * cols;
  T* yr = y + row * cols;
  float m = -INFINITY;
  for (int c = threadIdx.x; c < limit; c += blockDim.x) m = fmaxf(m, ldf(xr + c) * scale);
  m = block_reduce(m, red, true);
  const bool bad = !(fabsf(m) <= 3.0e38f);  // NaN or +-inf
  float s = 0.f;
  if (!bad)
    for (int c = threadIdx.x; c < limit; c += blockDim.x) s += __expf(ldf(xr + c) * scale - m);
  s = block_reduce(s, red, false);
  const float inv = (!bad && s > 0.f) ? 1.f / s : 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float v = (c < limit && inv > 0.f) ? __expf(ldf(xr + c) * scale - m) * inv : 0.f;
    stf(yr + c, v);
  }
}
// dx = scale * y * (dy - sum(dy*y))
__global__ void __launch_bounds__(256)
softmax_bwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ dy,
                   __nv_bfloat16* __restrict__ dx, int cols, float scale) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const __nv_bfloat16* yr = y + row * cols;
  const __nv_bfloat16* dr = dy + row * cols;
  float s = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x)
    s += __bfloat162float(yr[c]) * __bfloat162float(dr[c]);
  s = block_reduce(s, red, false);
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float p = __bfloat162float(yr[c]);
    dx[row * cols + c] = __float2bfloat16(scale * p * (__bfloat162float(dr[c]) - s));
  }
}

// ----------------------------------------------------------------------------- cross entropy
// One CTA per row.  The bf16 row is staged in shared memory when it fits, so the logits are read from HBM once
// and the gradient is written once (in place allowed).  The kernel is bound by instruction issue and by the
// exponential unit (two exponentials per logit), so both walks over the row are written for a short instruction
// stream: bf16 pairs are widened with one shift / mask each, every exponential is one FFMA into ex2.approx
// (log2(e) folded into the operands), and the vectors past the vocabulary are not visited by the first walk.
constexpr int CE_THREADS = 1024;
constexpr float CE_LOG2E = 1.4426950408889634f;
__device__ __forceinline__ float ce_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void ce_widen(const uint4& u, float* f) {
  f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
  f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
  f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
  f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}
__global__ void __launch_bounds__(CE_THREADS, 2)
cross_entropy_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
                     float* __restrict__ losses, __nv_bfloat16* __restrict__ dlogits, int vocab,
                     int ld, float grad_scale, int use_smem) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ uint4 ce_smem[];
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const __nv_bfloat16* xr = logits + row * ld;
  const uint4* xv = reinterpret_cast<const uint4*>(xr);
  const int nvec = ld >> 3;
  const int nfull = vocab >> 3;                 // vectors that lie wholly inside the vocabulary
  const int nvalid = (vocab + 7) >> 3;          // vectors that hold at least one logit
  const long long tgt = targets[row];
  // Online softmax statistics while the row streams in: each thread keeps a running maximum mt (in units of
  // log2, i.e. x * log2(e)) and the sum st of 2^(x' - mt) over its own vectors, rescaled when the maximum moves,
  // so the exponentials of the first walk run under the latency of the loads.
  float mt = -INFINITY, st = 0.f;
  auto absorb = [&](const uint4& u, int v) {
    float f[8];
    ce_widen(u, f);
    if (v >= nfull) {               // the one vector that straddles the end of the vocabulary: padding never counts
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (v * 8 + i >= vocab) f[i] = -INFINITY;
    }
    const float vm = fmaxf(fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3])), fmaxf(fmaxf(f[4], f[5]), fmaxf(f[6], f[7])));
    const float mn = fmaxf(mt, vm * CE_LOG2E);
    const float sc = (mt == mn) ? 1.f : ce_ex2(mt - mn);        // mt = -inf on the first vector: 2^-inf = 0
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      a0 += ce_ex2(fmaf(f[i], CE_LOG2E, -mn));
      a1 += ce_ex2(fmaf(f[i + 1], CE_LOG2E, -mn));
    }
    st = fmaf(st, sc, a0 + a1);
    mt = mn;
  };
  if (use_smem) {
    // The whole row is requested at once with 16-byte asynchronous copies straight into shared memory (no
    // registers hold data in flight), committed in groups of four per thread; each thread then waits for its
    // own groups in order and absorbs the vectors it copied itself, so no CTA barrier separates copy and use.
    const uint32_t sbase = smem_u32(ce_smem);
    int groups = 0;
    for (int v0 = threadIdx.x; v0 < nvalid; v0 += 4 * CE_THREADS) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = v0 + k * CE_THREADS;
        if (v < nvalid)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + 16u * v), "l"(xv + v) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      ++groups;
    }
    int g = 0;
    for (int v0 = threadIdx.x; v0 < nvalid; v0 += 4 * CE_THREADS, ++g) {
      switch (groups - 1 - g) {     // groups still allowed to be in flight
        case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = v0 + k * CE_THREADS;
        if (v < nvalid) absorb(ce_smem[v], v);
      }
    }
  } else {
    // rows too long for shared memory: four 16-byte loads in flight per thread, second walk re-reads from L2
    for (int v0 = threadIdx.x; v0 < nvalid; v0 += 4 * CE_THREADS) {
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = v0 + k * CE_THREADS;
        if (v < nvalid) u[k] = xv[v];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = v0 + k * CE_THREADS;
        if (v < nvalid) absorb(u[k], v);
      }
    }
  }
  const float m2 = block_reduce(mt, red, true);                  // row maximum times log2(e)
  // per-thread sums are brought to the common maximum and added in the fixed order of the block reduction
  const float s = block_reduce(mt == -INFINITY ? 0.f : st * ce_ex2(mt - m2), red, false);
  const uint4* src = use_smem ? ce_smem : xv;
  const bool ignore = !(tgt >= 0 && tgt < vocab);
  if (threadIdx.x == 0) {
    const float xt = ignore ? 0.f : __bfloat162float(use_smem ? reinterpret_cast<const __nv_bfloat16*>(ce_smem)[tgt] : xr[tgt]);
    losses[row] = ignore ? 0.f : (m2 + __log2f(s)) * 0.6931471805599453f - xt;
  }
  if (dlogits) {
    __syncthreads();  // the target logit was read before any in-place write
    uint4* ov = reinterpret_cast<uint4*>(dlogits + row * ld);
    if (ignore) {
      for (int v = threadIdx.x; v < nvec; v += CE_THREADS) ov[v] = make_uint4(0u, 0u, 0u, 0u);
      return;
    }
    const float k = grad_scale / s;                 // softmax normalisation and loss scale in one factor
    const int vt = (int)(tgt >> 3);                 // the vector that holds the target column
    for (int v = threadIdx.x; v < nvec; v += CE_THREADS) {
      if (v >= nvalid) {                            // padding columns carry no gradient
        ov[v] = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
      float f[8];
      ce_widen(src[v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = ce_ex2(fmaf(f[i], CE_LOG2E, -m2)) * k;
      if (v == vt || v >= nfull) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int c = v * 8 + i;
          if (c == tgt) f[i] -= grad_scale;
          if (c >= vocab) f[i] = 0.f;
        }
      }
      ov[v] = pack8(f);
    }
  }
}

// ----------------------------------------------------------------------------- reductions
// Single CTA, fixed tree: each thread sums a strided slice serially, then a fixed
// shuffle/shared tree combines the 1024 partials.  Result is independent of anything
// but n, so it replays bit-identically.
template <bool SQUARE>
__global__ void __launch_bounds__(1024)
reduce_one_block_kernel(const float* __restrict__ x, float* __restrict__ out, long long n,
                        float scale, int accumulate) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[33];
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += 1024) {
    float v = x[i];
    s += SQUARE ? v * v : v;
  }
  s = block_reduce(s, red, false);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s * scale : s * scale;
}
// Two-level version for large buffers: level 1 writes one partial per CTA.
template <bool SQUARE>
__global__ void __launch_bounds__(256)
reduce_level1_kernel(const float* __restrict__ x, float* __restrict__ partial, long long n) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[33];
  const long long per = (n + gridDim.x - 1) / gridDim.x;
  const long long b = per * blockIdx.x, e = (b + per < n) ? b + per : n;
  float s = 0.f;
  for (long long i = b + threadIdx.x; i < e; i += 256) {
    float v = x[i];
    s += SQUARE ? v * v : v;
  }
  s = block_reduce(s, red, false);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

}  // namespace ftk

using namespace ftk;
#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define BF(p) reinterpret_cast<const __nv_bfloat16*>(p)
#define BFW(p) reinterpret_cast<__nv_bfloat16*>(p)

template <bool RMS>
static int norm_fwd_launch(const void* x, const void* resid, void* sum_out, const void* gamma, const void* beta, void* y,
                           float* mean, float* rstd, int rows, int cols, float eps, cudaStream_t s) {
#define FT_NORM_FWD(NV, WPR, ...)                                                                              \
  launch_pdl(norm_fwd_kernel<NV, WPR, RMS, ##__VA_ARGS__>, WPR == 1 ? (rows + 3) / 4 : rows, WPR == 8 ? 256 : 128, 0, s,             \
      BF(x), BF(resid), BFW(sum_out), BF(gamma), BF(beta), BFW(y), mean, rstd, rows, cols, eps)
  const int nvec = cols / 8, per_lane = (nvec + 31) / 32;
  // Up to 1536 columns a row is one warp's.  Wider rows take a CTA each, except where there are enough rows of up to 2048
  // columns to fill the chip with warps (one / four / eight warps per row, RMS: 30000 x 2048 38.5 / 42.5 / - us, 8192 x 2048 9.9 / 10.1 /
  // -, 4096 x 2048 7.3 / 5.8 / -, 1500 x 2048 - / 3.3 / 3.6, 64 x 2048 - / 1.7 / 1.8).  2056 to 3072 columns are three vectors a lane of
  // four warps, where eight warps leave a quarter of the lanes idle (8192 x 3072: 19.5 against 27.4 us, RMS 17.0 against 20.5;
  // 500 x 3072 level, below that the wider CTA is quicker).  A row stays in registers up to 16384 columns: 8192 x 16384 107 us
  // against 226 walked three times by a warp, 1 x 16384 4.4 against 30.
  if (per_lane <= 1) FT_NORM_FWD(1, 1);
  else if (per_lane <= 2) FT_NORM_FWD(2, 1);
  else if (per_lane <= 3) FT_NORM_FWD(3, 1);
  else if (per_lane <= 4 && rows >= 4096) FT_NORM_FWD(4, 1, true);
  else if (per_lane <= 4) FT_NORM_FWD(4, 1);
  else if (per_lane <= 6) FT_NORM_FWD(6, 1);
  else if (per_lane <= 8 && rows >= 8192) FT_NORM_FWD(8, 1);
  else if (per_lane <= 8 && rows >= 500) FT_NORM_FWD(2, 4);
  else if (nvec <= 256) FT_NORM_FWD(1, 8);
  else if (nvec <= 384 && rows >= 500) FT_NORM_FWD(3, 4);
  else if (nvec <= 512) FT_NORM_FWD(2, 8);
  else if (nvec <= 1024) FT_NORM_FWD(4, 8);
  else if (nvec <= 2048) FT_NORM_FWD(8, 8);
  else
    launch_pdl(norm_fwd_long_kernel<RMS>, rows, ROW_WARPS * 32, 0, s,
        BF(x), BF(resid), BFW(sum_out), BF(gamma), BF(beta), BFW(y), mean, rstd, rows, cols, eps);
#undef FT_NORM_FWD
  return (int)cudaGetLastError();
}
extern "C" int ftk_layernorm_fwd(const void* x, const void* resid_in, void* sum_out,
                                 const void* gamma, const void* beta, void* y, float* mean,
                                 float* rstd, int rows, int cols, float eps, void* stream) {
  if (cols % 8 || rows <= 0) return -2;
  if (resid_in && !sum_out) return -3;
  return norm_fwd_launch<false>(x, resid_in, sum_out, gamma, beta, y, mean, rstd, rows, cols, eps, STREAM(stream));
}
extern "C" int ftk_rmsnorm_fwd(const void* x, const void* gamma, void* y, float* rstd, int rows,
                               int cols, float eps, void* stream) {
  if (cols % 8 || rows <= 0) return -2;
  return norm_fwd_launch<true>(x, nullptr, nullptr, gamma, nullptr, y, nullptr, rstd, rows, cols, eps, STREAM(stream));
}
// number of partial blocks the caller must provide room for (2 * blocks * cols floats)
static int norm_col_blocks(int rows) { return (rows + COL_ROWS_PER_BLK - 1) / COL_ROWS_PER_BLK; }
extern "C" int ftk_layernorm_bwd_blocks(int rows) {
  const int fused = rows < NB_MAX_BLOCKS ? rows : NB_MAX_BLOCKS, wide = norm_col_blocks(rows);
  return fused > wide ? fused : wide;
}

// One group where a single round of loads covers the partials, 8 groups up to two rounds, and for outputs that are wide enough
// to fill the chip with them; 32 groups for many partials of a narrow output.  Column sums in us, 32 / 8 / 1 groups:
// 500 x 8192 (8 partials) 6.5 / 5.0 / 4.0; 1500 x 3072 (24) 5.8 / 4.1 / 4.9; 8192 x 768 (128) 5.3 / 4.7 / 10.6; 8192 x 16384 56 / 51 / 60;
// 20000 x 768 (313) 7.8 / 8.2 / 23; LayerNorm backward 1500 x 3072 (296) 13.2 / 14.5 / 26, 1500 x 8192 30.9 / 29.2 / 45.
static int col_final(const float* partial, float* out, const float* partial2, float* out2, int cols, int nblk,
                     int accumulate, cudaStream_t s) {
  if (nblk <= 8)
    return launch_pdl(col_final_kernel<1>, (cols + 127) / 128, 128, 0, s, partial, out, partial2, out2, cols, nblk, accumulate);
  if (nblk <= 128 || cols >= 8192)
    return launch_pdl(col_final_kernel<8>, (cols + 31) / 32, 256, 0, s, partial, out, partial2, out2, cols, nblk, accumulate);
  return launch_pdl(col_final_kernel<32>, (cols + 31) / 32, 1024, 0, s, partial, out, partial2, out2, cols, nblk, accumulate);
}

template <int NV, int WPR, bool RMS>
static int norm_bwd_fused_launch(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd,
                                 const void* dx_add, void* dx, float* partial, int rows, int cols, int nblk, cudaStream_t s) {
  constexpr int G = ROW_WARPS / WPR;
  int* status = ftk_status_word();
  if (!status) return -6;
  const size_t stage = (size_t)(dx_add ? 3 : 2) * G * cols * 2;
  int stages = (int)(NB_RING_BYTES / stage);
  if (stages > 8) stages = 8;
  if (stages < 2) stages = 2;
  size_t smem = stages * stage;
  const size_t sums = G > 1 ? (size_t)(RMS ? 1 : 2) * G * cols * 4 : 0;
  if (smem < sums) smem = sums;
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(norm_bwd_fused_kernel<NV, WPR, RMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         112 * 1024);
    if (e != cudaSuccess) return (int)e;
    done[dev] = true;
  }
  launch_pdl(norm_bwd_fused_kernel<NV, WPR, RMS>, nblk, ROW_WARPS * 32, smem, s,
      BF(dy), BF(x), BF(gamma), mean, rstd, BF(dx_add), BFW(dx), partial, rows, cols, (rows + nblk - 1) / nblk, stages, status);
  return (int)cudaGetLastError();
}
template <bool RMS>
static int norm_bwd_launch(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd,
                           const void* dx_add, void* dx, float* dgamma, float* dbeta, float* partial, int rows, int cols,
                           int accumulate, cudaStream_t s) {
  const int nvec = cols / 8;
  int nblk = 0, rc = 0;
  // Tens of thousands of rows of a vector per lane or less: a warp per row in lock step with its CTA spends 1.4 us on a step of
  // eight, most of it latency, where the separate passes have all their warps in flight and find the rows in L2 again.  In us,
  // one pass / three kernels: RMS 8192 x 64 7.3 / 9.7, 30000 x 64 17.1 / 15.9, 65536 x 64 39.5 / 25.6, 65536 x 256 41.5 / 38.9,
  // 65536 x 384 48 / 79, 200000 x 128 115 / 101, 200000 x 256 116 / 129; LayerNorm 30000 x 64 19.4 / 19.8, 65536 x 64 45 / 32,
  // 65536 x 256 48 / 51 and with an added gradient 45 / 57, so 256 columns are for RMSNorm only.
  // (Row blocks ride on grid.y there.)
  const bool narrow = rows >= 24000 && norm_col_blocks(rows) <= 65535 &&
                      (nvec <= 16 || (RMS && nvec <= 32 && (long long)rows * cols <= 32ll << 20));
  if (dgamma && nvec <= 1024 && !narrow) {
    // One pass.  WPR warps per row so that a lane holds at most three vectors (four at the widest) and its column sums stay
    // in registers.
    const int wpr = nvec <= 96 ? 1 : (nvec <= 192 ? 2 : (nvec <= 384 ? 4 : 8));
    const int nv = (nvec + 32 * wpr - 1) / (32 * wpr), G = ROW_WARPS / wpr;
    nblk = (rows + G - 1) / G;
    if (nblk > NB_MAX_BLOCKS) nblk = NB_MAX_BLOCKS;
    const int per = ((rows + nblk - 1) / nblk + G - 1) / G * G;     // whole steps
    nblk = (rows + per - 1) / per;
#define FT_NORM_BWD(NV, WPR) \
  rc = norm_bwd_fused_launch<NV, WPR, RMS>(dy, x, gamma, mean, rstd, dx_add, dx, partial, rows, cols, nblk, s)
    switch (wpr * 8 + nv) {
      case 9: FT_NORM_BWD(1, 1); break;
      case 10: FT_NORM_BWD(2, 1); break;
      case 11: FT_NORM_BWD(3, 1); break;
      case 18: FT_NORM_BWD(2, 2); break;
      case 19: FT_NORM_BWD(3, 2); break;
      case 34: FT_NORM_BWD(2, 4); break;
      case 35: FT_NORM_BWD(3, 4); break;
      case 66: FT_NORM_BWD(2, 8); break;
      case 67: FT_NORM_BWD(3, 8); break;
      case 68: FT_NORM_BWD(4, 8); break;
      default: return -7;
    }
#undef FT_NORM_BWD
    if (rc) return rc;
  } else {
    launch_pdl(norm_bwd_dx_kernel<RMS>, (rows + ROW_WARPS - 1) / ROW_WARPS, ROW_WARPS * 32, 0, s,
        BF(dy), BF(x), BF(gamma), mean, rstd, BF(dx_add), BFW(dx), rows, cols);
    if (!dgamma) return (int)cudaGetLastError();
    nblk = norm_col_blocks(rows);
    dim3 g((cols / 2 + 31) / 32, nblk);
    launch_pdl(col_partial_kernel<RMS ? 1 : 0>, g, 256, 0, s, BF(dy), BF(x), mean, rstd, partial, rows, cols, cols, nblk);
  }
  col_final(partial, dgamma, RMS ? nullptr : partial + (size_t)nblk * cols, dbeta, cols, nblk, accumulate, s);
  return (int)cudaGetLastError();
}
extern "C" int ftk_layernorm_bwd(const void* dy, const void* x, const void* gamma,
                                 const float* mean, const float* rstd, const void* dx_add, void* dx,
                                 float* dgamma, float* dbeta, float* partial, int rows, int cols,
                                 int accumulate, void* stream) {
  if (cols % 8 || rows <= 0) return -2;
  return norm_bwd_launch<false>(dy, x, gamma, mean, rstd, dx_add, dx, dgamma, dbeta, partial, rows, cols, accumulate,
                                STREAM(stream));
}
extern "C" int ftk_rmsnorm_bwd(const void* dy, const void* x, const void* gamma, const float* rstd,
                               void* dx, float* dgamma, float* partial, int rows, int cols,
                               int accumulate, void* stream) {
  if (cols % 8 || rows <= 0) return -2;
  return norm_bwd_launch<true>(dy, x, gamma, nullptr, rstd, nullptr, dx, dgamma, nullptr, partial, rows, cols, accumulate,
                               STREAM(stream));
}
// Plain column sums with 16-byte loads: a CTA covers 256 columns x CSW_ROWS rows as 8 row groups of
// 32 lanes x 8 columns.  Each thread adds its rows (r0 + group, + 8, ...) in ascending order with four
// row loads in flight, then group 0 adds the 8 group sums in group order: a fixed tree again.
constexpr int CSW_ROWS = 64;
__global__ void __launch_bounds__(256)
colsum_wide_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ partial, int rows, int cols,
                   long long ld) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sm[COL_GROUPS][32][9];
  const int lane = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * 8;
  const int blk = blockIdx.y;
  const int r0 = blk * CSW_ROWS;
  const int r1 = min(rows, r0 + CSW_ROWS);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < cols) {
    int r = r0 + rg;
    for (; r + 3 * COL_GROUPS < r1; r += 4 * COL_GROUPS) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = __ldg(reinterpret_cast<const uint4*>(x + (size_t)(r + u * COL_GROUPS) * ld + c));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 f0 = unpack_bf16(v[u].x), f1 = unpack_bf16(v[u].y), f2 = unpack_bf16(v[u].z),
                     f3 = unpack_bf16(v[u].w);
        acc[0] += f0.x; acc[1] += f0.y; acc[2] += f1.x; acc[3] += f1.y;
        acc[4] += f2.x; acc[5] += f2.y; acc[6] += f3.x; acc[7] += f3.y;
      }
    }
    for (; r < r1; r += COL_GROUPS) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(x + (size_t)r * ld + c));
      const float2 f0 = unpack_bf16(w.x), f1 = unpack_bf16(w.y), f2 = unpack_bf16(w.z), f3 = unpack_bf16(w.w);
      acc[0] += f0.x; acc[1] += f0.y; acc[2] += f1.x; acc[3] += f1.y;
      acc[4] += f2.x; acc[5] += f2.y; acc[6] += f3.x; acc[7] += f3.y;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) sm[rg][lane][i] = acc[i];
  __syncthreads();
  if (rg == 0 && c < cols) {
    float t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = 0.f;
#pragma unroll
    for (int k = 0; k < COL_GROUPS; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] += sm[k][lane][i];
    float* dst = partial + (size_t)blk * cols + c;
    reinterpret_cast<float4*>(dst)[0] = make_float4(t[0], t[1], t[2], t[3]);
    reinterpret_cast<float4*>(dst)[1] = make_float4(t[4], t[5], t[6], t[7]);
  }
}

// Number of row blocks (= rows of the partial buffer the caller provides) for `rows` input rows.
extern "C" int ftk_colsum_blocks(int rows) { return (rows + CSW_ROWS - 1) / CSW_ROWS; }

extern "C" int ftk_colsum_bf16(const void* x, float* out, float* partial, int rows, int cols,
                               long long ld, int accumulate, void* stream) {
  if (cols % 2 || ld % 2 || rows <= 0) return -2;
  cudaStream_t s = STREAM(stream);
  const bool wide = (cols % 8 == 0) && (ld % 8 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0) &&
                    ((reinterpret_cast<uintptr_t>(partial) & 15) == 0);
  int nblk;
  if (wide) {
    nblk = ftk_colsum_blocks(rows);
    dim3 g((cols / 8 + 31) / 32, nblk);
    launch_pdl(colsum_wide_kernel, g, 256, 0, s, BF(x), partial, rows, cols, ld);
  } else {
    // odd extents / alignments: two columns per thread; needs fewer row blocks than were provided for
    nblk = (rows + COL_ROWS_PER_BLK - 1) / COL_ROWS_PER_BLK;
    dim3 g((cols / 2 + 31) / 32, nblk);
    launch_pdl(col_partial_kernel<2>, g, 256, 0, s, BF(x), nullptr, nullptr, nullptr, partial, rows, cols, ld, nblk);
  }
  col_final(partial, out, nullptr, nullptr, cols, nblk, accumulate, s);
  return (int)cudaGetLastError();
}

extern "C" int ftk_softmax_rows(const void* x, void* y, int rows, int cols, int is_bf16,
                                void* stream) {
  if (rows <= 0 || cols <= 0) return -2;
  if (is_bf16)
    launch_pdl(softmax_rows_kernel<__nv_bfloat16>, rows, 256, 0, STREAM(stream), BF(x), BFW(y), cols, 0, 1.f);
  else
    launch_pdl(softmax_rows_kernel<float>, rows, 256, 0, STREAM(stream),
        reinterpret_cast<const float*>(x), reinterpret_cast<float*>(y), cols, 0, 1.f);
  return (int)cudaGetLastError();
}
extern "C" int ftk_softmax_causal_bf16(const void* x, void* y, int L, int S, float scale,
                                       void* stream) {
  if (L <= 0 || S <= 0) return -2;
  launch_pdl(softmax_rows_kernel<__nv_bfloat16>, (unsigned)((size_t)L * S), 256, 0, STREAM(stream),
      BF(x), BFW(y), S, S, scale);
  return (int)cudaGetLastError();
}
extern "C" int ftk_softmax_bwd_bf16(const void* y, const void* dy, void* dx, long long rows,
                                    int cols, float scale, void* stream) {
  if (rows <= 0 || cols <= 0) return -2;
  launch_pdl(softmax_bwd_kernel, (unsigned)rows, 256, 0, STREAM(stream), BF(y), BF(dy), BFW(dx), cols, scale);
  return (int)cudaGetLastError();
}

extern "C" int ftk_cross_entropy_fwd_bwd(const void* logits, const long long* targets,
                                         float* losses, void* dlogits, int rows, int vocab, int ld,
                                         float grad_scale, void* stream) {
  if (ld % 8 || vocab > ld || rows <= 0) return -2;
  const size_t bytes = (size_t)ld * 2;
  const int use_smem = bytes <= 200 * 1024;     // longer rows are re-read from L2 by the second walk
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(cross_entropy_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  launch_pdl(cross_entropy_kernel, rows, CE_THREADS, use_smem ? bytes : 0, STREAM(stream),
      BF(logits), targets, losses, BFW(dlogits), vocab, ld, grad_scale, use_smem);
  return (int)cudaGetLastError();
}

extern "C" int ftk_reduce_mean_f32(const float* x, float* out, long long n, float scale,
                                   void* stream) {
  if (n <= 0) return -2;
  launch_pdl(reduce_one_block_kernel<false>, 1, 1024, 0, STREAM(stream), x, out, n, scale, 0);
  return (int)cudaGetLastError();
}
extern "C" int ftk_sumsq_f32(const float* x, float* out, float* partial, long long n,
                             int accumulate, void* stream) {
  if (n <= 0) return -2;
  if (n < (1 << 16) || !partial) {
    launch_pdl(reduce_one_block_kernel<true>, 1, 1024, 0, STREAM(stream), x, out, n, 1.f, accumulate);
  } else {
    // level 1: FTK_SUMSQ_PARTIALS fixed slices; level 2: one block over the partials
    launch_pdl(reduce_level1_kernel<true>, FTK_SUMSQ_PARTIALS, 256, 0, STREAM(stream), x, partial, n);
    launch_pdl(reduce_one_block_kernel<false>, 1, 1024, 0, STREAM(stream), partial, out, FTK_SUMSQ_PARTIALS,
                                                                    1.f, accumulate);
  }
  return (int)cudaGetLastError();
}
