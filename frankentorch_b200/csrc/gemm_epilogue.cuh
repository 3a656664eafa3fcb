// Epilogue of the sm_100a GEMMs: one warp turns its 32-row slab of an accumulator tile into output.
//
// A thread owns one accumulator row (that is how tcgen05.ld delivers it), while global memory wants 64 or 128
// contiguous bytes of a row per group of lanes.  Everything row-shaped (residual / activation operand in,
// pre-activation and output out) therefore crosses a 4 KB shared-memory tile of the warp, 32 columns at a time,
// 16-byte segments XOR-swizzled so that both directions are free of bank conflicts.  The bias of the warp's columns is
// brought into shared memory and the first residual chunk into registers before the accumulator is waited for, the next
// residual chunk while the current one is processed, so no chunk starts with a global-memory round trip.
//
// What bounds it: the issue slots and the tanh unit of two warps per scheduler (a 32-column chunk takes ~700 cycles
// plain, ~1400 with GELU and the pre-activation) against the main loop of the next tile.  With scalar bias loads and
// per-row residual / pre-activation accesses in one body for all kinds a chunk took ~1900 and ~4000 cycles:
// 32 x 2048 x 512 with bias 11.3 -> 5.1 us, 8192 x 3072 x 768 with bias, GELU and pre-activation 75.3 -> 39.7 us, with GELU'
// of a residual operand 66.3 -> 42.0 us (both together with the issue loops of the kernels, see mbar_wait_warp).
//
// Outputs and operands whose extents or alignment do not allow 16-byte segments take the general path: the chunk goes to
// the tile in fp32 and is written row by row, lane = column, eight rows at a time.
#pragma once
#include "ft_sm100.cuh"
#include "ftk_api.h"
#include "launch.cuh"

namespace ftk {

constexpr int EPI_STAGE_BYTES = 4096;   // per warp
constexpr int EPI_BIAS_BYTES = 256;     // per warp: 128 bf16

struct GemmArgs {
  int M, N, K, L0, L1;
  int a_mn, b_mn;
  void* D;
  long long ldd, d_s0, d_s1;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* resid;
  long long ldr, r_s0, r_s1;
  __nv_bfloat16* aux;  // optional bf16 copy of the pre-activation (same layout as D)
  float alpha;
  int epi;
  int out_fp32;
  int accumulate;
  int splits;          // >1: split-K, partial tiles go to `ws` as fp32 [split][M][N]
  float* ws;
  int* status;
  // Ragged rows (expert batches): the M rows of batch l are segments of `seg_rows` rows of which
  // only the first seg_counts[l * segs + s] are in use; a 128-row tile without a used row is
  // skipped by every role (no loads, no MMAs, no stores).  NULL = all rows in use.
  const int* seg_counts;
  int seg_rows;
  // work item = ((split * batches + batch) * n tiles + n tile) * m tiles + m tile; pair tiles take the m tiles in groups of
  // by_gm.d (the last group by_gm_last.d) that walk all n tiles
  FastDiv by_tiles_m, by_tiles_mn, by_batches, by_l0, by_group, by_gm, by_gm_last;
};

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Epilogue activations use the hardware tanh (relative error ~2^-11, below bf16 rounding).
__device__ __forceinline__ float gelu_tanh_fast(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.f + tanh_fast(u));
}
__device__ __forceinline__ float gelu_tanh_grad_fast(float x) {
  const float x2 = x * x;
  const float t = tanh_fast(0.7978845608028654f * (x + 0.044715f * x * x2));
  const float du = 0.7978845608028654f * (1.f + 3.f * 0.044715f * x2);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}

// One value through the activation: `r` is the operand of the MUL_* forms.
__device__ __forceinline__ float apply_epi(float v, float r, int epi) {
  switch (epi) {
    case FTK_EPI_GELU_TANH: return gelu_tanh_fast(v);
    case FTK_EPI_GELU_ERF: return gelu_erf_f(v);
    case FTK_EPI_RELU: return v > 0.f ? v : 0.f;
    case FTK_EPI_MUL_DGELU_TANH: return v * gelu_tanh_grad_fast(r);
    case FTK_EPI_MUL_DGELU_ERF: return v * gelu_erf_grad_f(r);
    case FTK_EPI_MUL_DRELU: return r > 0.f ? v : 0.f;
    default: return v;
  }
}
// The two tanh-form activations on pairs: 5 and 9 packed operations instead of 12 and 24 scalar ones per pair.
__device__ __forceinline__ f32x2 gelu_tanh2(f32x2 x) {
  const f32x2 x2 = mul2(x, x);
  const f32x2 u = mul2(x, fma2(x2, pk2(0.035677408136300125f, 0.035677408136300125f),
                               pk2(0.7978845608028654f, 0.7978845608028654f)));
  const float2 us = up2(u);
  const f32x2 h = mul2(x, pk2(0.5f, 0.5f));
  return fma2(h, pk2(tanh_fast(us.x), tanh_fast(us.y)), h);
}
__device__ __forceinline__ f32x2 gelu_tanh_grad2(f32x2 x) {
  const f32x2 k0 = pk2(0.7978845608028654f, 0.7978845608028654f), half = pk2(0.5f, 0.5f);
  const f32x2 x2 = mul2(x, x);
  const float2 us = up2(mul2(x, fma2(x2, pk2(0.035677408136300125f, 0.035677408136300125f), k0)));
  const f32x2 t = pk2(tanh_fast(us.x), tanh_fast(us.y));
  const f32x2 du = fma2(x2, pk2(0.10703222440890037f, 0.10703222440890037f), k0);
  const f32x2 omt2 = fma2(mul2(t, pk2(-1.f, -1.f)), t, pk2(1.f, 1.f));
  return fma2(mul2(mul2(x, half), omt2), du, fma2(half, t, half));
}
// The same for the 32 values of one row chunk, the switch outside the loop; `rp` holds the operand as bf16 pairs.
__device__ __forceinline__ void apply_epi32(f32x2* v, const uint32_t* rp, int epi) {
#define FT_EPI_LOOP(expr)                                       \
  _Pragma("unroll") for (int i = 0; i < 16; ++i) {              \
    const float2 x = up2(v[i]), r = unpack_bf16(rp[i]);         \
    (void)x; (void)r;                                           \
    v[i] = (expr);                                              \
  }
  switch (epi) {
    case FTK_EPI_GELU_TANH: FT_EPI_LOOP(gelu_tanh2(v[i])) break;
    case FTK_EPI_GELU_ERF: FT_EPI_LOOP(pk2(gelu_erf_f(x.x), gelu_erf_f(x.y))) break;
    case FTK_EPI_RELU: FT_EPI_LOOP(pk2(x.x > 0.f ? x.x : 0.f, x.y > 0.f ? x.y : 0.f)) break;
    case FTK_EPI_MUL_DGELU_TANH: FT_EPI_LOOP(mul2(v[i], gelu_tanh_grad2(pk2(r.x, r.y)))) break;
    case FTK_EPI_MUL_DGELU_ERF: FT_EPI_LOOP(pk2(x.x * gelu_erf_grad_f(r.x), x.y * gelu_erf_grad_f(r.y))) break;
    case FTK_EPI_MUL_DRELU: FT_EPI_LOOP(pk2(r.x > 0.f ? x.x : 0.f, r.y > 0.f ? x.y : 0.f)) break;
    default: break;
  }
#undef FT_EPI_LOOP
}

// Epilogue kinds.  The ones that training and inference use have their own instantiation (no run-time switches, no
// registers held for parts they lack; with everything in one body a plain 32-column chunk took 900 cycles);
// EPI_KIND_ANY takes every other combination and every alignment.
enum : int {
  EPI_KIND_ANY = 0,
  EPI_KIND_PLAIN = 1,      // bf16 out (+ bias)
  EPI_KIND_RESID = 2,      // bf16 out (+ bias) + residual
  EPI_KIND_GELU = 3,       // bf16 out, tanh GELU (+ bias)
  EPI_KIND_GELU_AUX = 4,   // the same, pre-activation kept
  EPI_KIND_DGELU = 5,      // bf16 out, times tanh GELU' of the operand
  EPI_KIND_F32 = 6,        // fp32 out (accumulating or not), or split-K partials
};

template <int KIND>
struct TileEpilogue {
  static constexpr bool ANY = KIND == EPI_KIND_ANY;
  static constexpr bool CAN_R = ANY || KIND == EPI_KIND_RESID || KIND == EPI_KIND_DGELU;
  static constexpr bool CAN_AUX = ANY || KIND == EPI_KIND_GELU_AUX;
  static constexpr bool CAN_BIAS = KIND != EPI_KIND_DGELU && KIND != EPI_KIND_F32;
  static constexpr bool CAN_F32 = ANY || KIND == EPI_KIND_F32;
  static constexpr bool CAN_BF16 = KIND != EPI_KIND_F32;
  enum : int { SLOW = 0, BF16 = 1, F32 = 2 };
  const GemmArgs& p;
  uint8_t* stage;
  __nv_bfloat16* sbias;
  int lane;
  // of the current tile
  int mode_, row0, n_base;
  bool empty_split;
  void* d;                       // row `row0`, column 0 of the destination
  long long ldd_;
  const __nv_bfloat16* resid;    // row `row0`, column 0
  __nv_bfloat16* aux;
  bool r_vec_;                   // the residual's rows are whole 16-byte segments
  uint32_t rw[16];               // residual chunk in flight: words 4 i .. of row 8 i + lane / 4, segment lane % 4, or
                                 // (rows that are not whole segments) column `lane` of rows 2 i and 2 i + 1

  __device__ __forceinline__ TileEpilogue(const GemmArgs& args, uint8_t* st, __nv_bfloat16* sb, int ln)
      : p(args), stage(st), sbias(sb), lane(ln) {}

  __device__ __forceinline__ bool split() const { return CAN_F32 && p.splits > 1; }
  __device__ __forceinline__ bool has_r() const { return CAN_R && (!ANY || (p.resid != nullptr && !split())); }
  __device__ __forceinline__ bool has_aux() const { return CAN_AUX && (!ANY || (p.aux != nullptr && !split())); }
  __device__ __forceinline__ bool has_bias() const { return CAN_BIAS && p.bias != nullptr && !split(); }
  __device__ __forceinline__ int mode() const { return ANY ? mode_ : (CAN_F32 ? F32 : BF16); }
  __device__ __forceinline__ long long ldd() const { return CAN_F32 ? ldd_ : p.ldd; }
  __device__ __forceinline__ int epi() const {
    if (KIND == EPI_KIND_GELU || KIND == EPI_KIND_GELU_AUX) return FTK_EPI_GELU_TANH;
    if (KIND == EPI_KIND_DGELU) return FTK_EPI_MUL_DGELU_TANH;
    return ANY ? p.epi : FTK_EPI_NONE;
  }

  // Rows [row, row + 32), columns from `col` on, `chunks` (<= 4) chunks of 32 columns, of (split sp, batch l).
  __device__ __forceinline__ void begin(int sp, int l, int row, int col, int chunks, bool empty) {
    row0 = row;
    n_base = col;
    empty_split = empty;
    const int l1 = p.by_l0.div(l), l0 = l - l1 * p.L0;
    if (split()) {
      d = p.ws + (((long long)sp * (p.L0 * p.L1) + l) * p.M + row) * p.N;
      ldd_ = p.N;
      mode_ = (p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(p.ws) & 15) == 0) ? F32 : SLOW;
      return;
    }
    const long long off = l0 * p.d_s0 + l1 * p.d_s1 + (long long)row * p.ldd;
    const int es = (CAN_F32 && (!CAN_BF16 || p.out_fp32)) ? 4 : 2;
    d = reinterpret_cast<uint8_t*>(p.D) + off * es;
    ldd_ = p.ldd;
    if (CAN_AUX) aux = p.aux + off;
    if (CAN_R) resid = p.resid + l0 * p.r_s0 + l1 * p.r_s1 + (long long)row * p.ldr;
    if (ANY) {
      bool ok = ((reinterpret_cast<uintptr_t>(d) & 15) == 0) && p.ldd % (16 / es) == 0 && p.N % (16 / es) == 0;
      r_vec_ = ((reinterpret_cast<uintptr_t>(resid) & 15) == 0) && p.ldr % 8 == 0 && p.N % 8 == 0;
      if (has_aux()) ok = ok && !p.out_fp32 && ((reinterpret_cast<uintptr_t>(aux) & 15) == 0);
      if (p.accumulate && !p.out_fp32) ok = false;
      mode_ = !ok ? SLOW : (p.out_fp32 ? F32 : BF16);
    }
    if (has_bias()) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < chunks) {
          const int c = col + 32 * j + lane;
          sbias[32 * j + lane] = c < p.N ? p.bias[c] : __float2bfloat16(0.f);
        }
      __syncwarp();
    }
    if (has_r() && mode() != SLOW) fetch_resid(col);
  }
  __device__ __forceinline__ bool r_vec() const { return !ANY || r_vec_; }
  // Rows that are not whole 16-byte segments come in 2 bytes per lane, 64 contiguous bytes of a row per warp, and leave the
  // output on the staged path (8192 x 768 x 3072 with residual rows of 8 bytes 114 us on the general path, 39 so).
  // (plain loads: the residual may be the output itself)
  __device__ __forceinline__ void fetch_resid(int n0) {
    if (r_vec()) {
      const int c = n0 + (lane & 3) * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        const uint4 u = (row0 + r < p.M && c < p.N) ? *reinterpret_cast<const uint4*>(resid + (long long)r * p.ldr + c)
                                                    : make_uint4(0u, 0u, 0u, 0u);
        rw[4 * i] = u.x; rw[4 * i + 1] = u.y; rw[4 * i + 2] = u.z; rw[4 * i + 3] = u.w;
      }
    } else {
      const unsigned short* rp = reinterpret_cast<const unsigned short*>(resid) + n0 + lane;
      const int rows = n0 + lane < p.N ? p.M - row0 : 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t lo = 2 * i < rows ? rp[(2 * i) * p.ldr] : 0, hi = 2 * i + 1 < rows ? rp[(2 * i + 1) * p.ldr] : 0;
        rw[i] = lo | (hi << 16);
      }
    }
  }
  // the fetched chunk into the tile
  __device__ __forceinline__ void put_resid() const {
    if (r_vec()) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *seg64(0, 8 * i + (lane >> 2), lane & 3) = make_uint4(rw[4 * i], rw[4 * i + 1], rw[4 * i + 2], rw[4 * i + 3]);
    } else {
#pragma unroll
      for (int r = 0; r < 32; ++r)
        reinterpret_cast<unsigned short*>(seg64(0, r, lane >> 3))[lane & 7] = (unsigned short)(rw[r >> 1] >> (16 * (r & 1)));
    }
  }
  // 64-byte rows: segment s (16 bytes) of row r
  __device__ __forceinline__ uint4* seg64(int half, int r, int s) const {
    return reinterpret_cast<uint4*>(stage + half * 2048 + r * 64 + ((s ^ ((r >> 1) & 3)) << 4));
  }
  // 128-byte rows
  __device__ __forceinline__ float4* seg128(int r, int s) const {
    return reinterpret_cast<float4*>(stage + r * 128 + ((s ^ (r & 7)) << 4));
  }
  __device__ __forceinline__ static uint32_t pack(f32x2 a) {
    const float2 f = up2(a);
    return pack_bf16(f.x, f.y);
  }
  __device__ __forceinline__ void put64(int half, const f32x2* v) const {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *seg64(half, lane, i) = make_uint4(pack(v[4 * i]), pack(v[4 * i + 1]), pack(v[4 * i + 2]), pack(v[4 * i + 3]));
  }
  __device__ __forceinline__ void store64(int half, __nv_bfloat16* dst, int n0) const {
    const int s = lane & 3, c = n0 + s * 8;
    __nv_bfloat16* dp = dst + (long long)(lane >> 2) * p.ldd + c;
    const int left = c < p.N ? p.M - row0 - (lane >> 2) : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 o = *seg64(half, 8 * i + (lane >> 2), s);
      if (8 * i < left) *reinterpret_cast<uint4*>(dp) = o;
      dp += 8 * p.ldd;
    }
  }
  __device__ __forceinline__ void store128(int n0) const {
    const int s = lane & 7, c = n0 + s * 4;
    float* dp = reinterpret_cast<float*>(d) + (long long)(lane >> 3) * ldd() + c;
    const int left = c < p.N ? p.M - row0 - (lane >> 3) : 0;
    const bool add = p.accumulate && !split();
    float4 old[8];
    if (add) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        old[i] = 4 * i < left ? *reinterpret_cast<const float4*>(dp + 4 * i * ldd()) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float4 o = *seg128(4 * i + (lane >> 3), s);
      if (add) {
        o.x += old[i].x; o.y += old[i].y; o.z += old[i].z; o.w += old[i].w;
      }
      if (4 * i < left) *reinterpret_cast<float4*>(dp) = o;
      dp += 4 * ldd();
    }
  }
  __device__ __forceinline__ void put128(const f32x2* v) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 a = up2(v[2 * i]), b = up2(v[2 * i + 1]);
      *seg128(lane, i) = make_float4(a.x, a.y, b.x, b.y);
    }
  }
  // General path, lane = column: the chunk is in the tile as scaled fp32, `bias` not yet added.
  __device__ __forceinline__ void store_general(int j, int n0) const {
    const int c = n0 + lane;
    const bool live = c < p.N;
    const float b = has_bias() ? __bfloat162float(sbias[32 * j + lane]) : 0.f;
    const int rows = min(32, p.M - row0);
    if (!live) return;
    // Eight rows at a time, all that is read of them requested before the first is written: row by row, each waits for its
    // own load (8192 x 769 x 3072 with bias and residual 146 -> 87 us, with fp32 accumulation 170 -> 87).
    const bool add = p.accumulate && !split();
#pragma unroll 1
    for (int r0 = 0; r0 < rows; r0 += 8) {
      float rr[8], old[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = r0 + k;
        rr[k] = old[k] = 0.f;
        if (has_r() && r < rows) rr[k] = __bfloat162float(resid[(long long)r * p.ldr + c]);
        if (add && r < rows)
          old[k] = p.out_fp32 ? reinterpret_cast<const float*>(d)[(long long)r * ldd() + c]
                              : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(d)[(long long)r * ldd() + c]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = r0 + k;
        if (r >= rows) break;
        float v = reinterpret_cast<const float*>(seg128(r, lane >> 2))[lane & 3] + b;
        const long long at = (long long)r * ldd() + c;
        if (split()) {
          reinterpret_cast<float*>(d)[at] = v;
          continue;
        }
        if (has_aux()) aux[at] = __float2bfloat16(v);
        v = apply_epi(v, rr[k], p.epi);
        if (has_r() && p.epi < FTK_EPI_MUL_DGELU_TANH) v += rr[k];
        if (add) v += old[k];
        if (p.out_fp32)
          reinterpret_cast<float*>(d)[at] = v;
        else
          reinterpret_cast<__nv_bfloat16*>(d)[at] = __float2bfloat16(v);
      }
    }
  }
  // Chunks [0, chunks) of the warp's columns, the accumulator at `tmem` (lane quarter included).  `release` runs once
  // the last chunk has been copied to registers.
  template <class Release>
  __device__ __forceinline__ void run(uint32_t tmem, int chunks, Release release) {
#pragma unroll 1
    for (int j = 0; j < chunks; ++j) {
      const int n0 = n_base + 32 * j;
      uint32_t acc[32];
      tmem_ld32(tmem + 32 * j, acc);
      uint32_t rp[16];
      if (has_r() && mode() != SLOW) {
        // residual: registers -> tile -> the row's own thread
        put_resid();
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 u = *seg64(0, lane, i);
          rp[4 * i] = u.x; rp[4 * i + 1] = u.y; rp[4 * i + 2] = u.z; rp[4 * i + 3] = u.w;
        }
        if (j + 1 < chunks) fetch_resid(n0 + 32);
        if (mode() == F32) __syncwarp();          // 128-byte rows overlap the neighbours' operand
      } else if (CAN_R) {
#pragma unroll
        for (int i = 0; i < 16; ++i) rp[i] = 0u;
      }
      tmem_ld_wait();
      if (j + 1 == chunks) release();
      f32x2 v[16];
      if (CAN_F32 && empty_split) {
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0u;
      }
      const f32x2 alpha = pk2(p.alpha, p.alpha);
      if (has_bias() && mode() != SLOW) {
        const uint4* sb = reinterpret_cast<const uint4*>(sbias + 32 * j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 u = sb[i];
          const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 b = unpack_bf16(w[k]);
            v[4 * i + k] = fma2(pk2(__uint_as_float(acc[8 * i + 2 * k]), __uint_as_float(acc[8 * i + 2 * k + 1])), alpha,
                                pk2(b.x, b.y));
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          v[i] = mul2(pk2(__uint_as_float(acc[2 * i]), __uint_as_float(acc[2 * i + 1])), alpha);
      }
      if (ANY && mode() == SLOW) {
        put128(v);
        __syncwarp();
        store_general(j, n0);
        __syncwarp();
        continue;
      }
      if (has_aux()) put64(1, v);
      if (!split()) {
        apply_epi32(v, rp, epi());
        if (has_r() && epi() < FTK_EPI_MUL_DGELU_TANH) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 r2 = unpack_bf16(rp[i]);
            v[i] = add2(v[i], pk2(r2.x, r2.y));
          }
        }
      }
      if (mode() == F32) {
        put128(v);
        __syncwarp();
        store128(n0);
      } else {
        put64(0, v);
        __syncwarp();
        if (has_aux()) store64(1, aux, n0);
        store64(0, reinterpret_cast<__nv_bfloat16*>(d), n0);
      }
      __syncwarp();
    }
  }
};

}  // namespace ftk
