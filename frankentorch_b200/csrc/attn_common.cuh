// Shared pieces of the sm_100a attention kernels: argument block, tcgen05 MMA helpers for the
// two operand forms used by attention, the swizzled probability-tile store, TMA tile loads and
// the host-side tensor-map construction over packed [B, S, H, hd] activations.
#pragma once
#include "ft_sm100.cuh"
#include "ftk_api.h"
#include "launch.cuh"

namespace ftk {

int ftk_make_tmap_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                       uint64_t l0, uint64_t l1, uint64_t ld_elems, uint64_t s0_elems,
                       uint64_t s1_elems, uint32_t box_inner, uint32_t box_outer);

constexpr int AT_T = 128;           // tile rows (queries) == tile keys
constexpr int AT_REGION = 16384;    // one [128 rows x 64 bf16] swizzled region

struct AttnArgs {
  int B, H, S;
  int causal;
  float sl2;    // scale * log2(e)
  float scale;
  const __nv_bfloat16* o;      // read by the dQ kernel (outputs leave through tensor maps)
  long long o_bs, o_ss, o_hs;
  float* lse;
  float* delta;             // written by the dQ kernel, read by the dK / dV kernel
  // Nothing reads these 96 bytes.  Without them the compiler allocates the registers of the backward loops of head size 64 another
  // way (dK / dV spills 8 bytes, dQ takes 83 instead of 85): B1 S4096 H6 causal 65.4 -> 67.5 us, B8 S256 H12 causal 14.9 -> 14.5.
  long long unused[12];
  int* status;
  int n_tiles;             // work items of the persistent kernels: blocks of rows x heads x batch
  FastDiv by_hb, by_h;     // / (H * B), / H
};

// Work items of one persistent CTA.  Items are numbered heaviest first (most blocks to visit under a causal mask); round r
// of the walk hands out gridDim.x of them, forwards in even rounds and backwards in odd ones, so that the CTA with the
// heaviest item of one round gets the lightest of the next.  Fixed by the grid: no counters, the same on every run.
struct TileWalk {
  int r, n;
  __device__ __forceinline__ explicit TileWalk(int n_items) : r(0), n(n_items) {}
  __device__ __forceinline__ int next() {
    const int G = (int)gridDim.x, c = (int)blockIdx.x;
    const int idx = r * G + ((r & 1) ? G - 1 - c : c);
    ++r;
    return idx < n ? idx : -1;
  }
};
// Ring position: slot and phase parity of the n-th use.
template <int N>
struct Ring {
  int s;
  uint32_t ph;
  __device__ __forceinline__ Ring() : s(0), ph(0) {}
  __device__ __forceinline__ void step() {
    if (++s == N) {
      s = 0;
      ph ^= 1u;
    }
  }
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 lanes of exp2, on the special-function unit.
__device__ __forceinline__ f32x2 exp2_pair(f32x2 x) {
  const float2 f = up2(x);
  return pk2(fast_exp2(f.x), fast_exp2(f.y));
}
__device__ __forceinline__ uint32_t pack2(f32x2 a) {
  const float2 f = up2(a);
  return pack_bf16(f.x, f.y);
}
__device__ __forceinline__ f32x2 acc2(const uint32_t* r, int i) {
  return pk2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
}

// A (K-major) x B (K-major)^T with K = HD, operands stored as HD/64 regions.  The descriptors'
// low words are built once per call and stepped by constants (see desc_lo).
template <int HD>
__device__ __forceinline__ void mma_kmajor(uint32_t d_tmem, uint32_t a_base, uint32_t b_base,
                                           uint32_t idesc) {
  const uint32_t a_lo = desc_lo(a_base, 16), b_lo = desc_lo(b_base, 16);
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    const uint32_t off = (uint32_t)(((kk >> 2) * AT_REGION + (kk & 3) * 32) >> 4);
    umma_bf16_lo(d_tmem, a_lo + off, b_lo + off, idesc, kk != 0 ? 1u : 0u);
  }
}
// A = probabilities [128 x 128] K-major in two regions; B = [128 k-rows x HD] stored
// row-major per 64-column region (MN-major operand), K = 128.
__device__ __forceinline__ void mma_p_times_rows(uint32_t d_tmem, uint32_t p_base, uint32_t b_base,
                                                 uint32_t idesc, bool accumulate) {
  const uint32_t a_lo = desc_lo(p_base, 16), b_lo = desc_lo(b_base, AT_REGION);
#pragma unroll
  for (int kk = 0; kk < AT_T / 16; ++kk) {
    const uint32_t a_off = (uint32_t)(((kk >> 2) * AT_REGION + (kk & 3) * 32) >> 4);
    umma_bf16_lo(d_tmem, a_lo + a_off, b_lo + (uint32_t)(kk * 128), idesc, (accumulate || kk != 0) ? 1u : 0u);
  }
}
// Same product with A = probabilities held in tensor memory: 128 lanes (rows) x 64 columns of
// packed bf16 pairs (K = 128), written by the row-owning threads with tcgen05.st.
// K steps [K0, K1) of 16.
template <int K0 = 0, int K1 = AT_T / 16>
__device__ __forceinline__ void mma_ptmem_times_rows(uint32_t d_tmem, uint32_t p_tmem, uint32_t b_base,
                                                     uint32_t idesc, bool accumulate) {
  const uint32_t b_lo = desc_lo(b_base, AT_REGION);
#pragma unroll
  for (int kk = K0; kk < K1; ++kk) {
    umma_bf16_ts_lo(d_tmem, p_tmem + kk * 8, b_lo + (uint32_t)(kk * 128), idesc,
                    (accumulate || kk != 0) ? 1u : 0u);
  }
}
template <int HD>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar,
                                          int row0, int h, int b) {
#pragma unroll
  for (int c = 0; c < HD / 64; ++c) tma_load_4d(dst + c * AT_REGION, tm, bar, c * 64, row0, h, b);
}


// ------------------------------------------------------------------------------- host helpers
// Boxes of `cols` x `rows`: the tiles that are loaded, or what a warp stores (32 columns: 64-byte swizzle).
static inline int make_map(CUtensorMap* m, const void* base, const FtkAttnDesc* a, long long bs,
                    long long ss, long long hs, unsigned cols = 64, unsigned rows = AT_T) {
  // dims {hd, S, H, B}; strides in elements
  typedef CUresult (*Fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                         const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                         CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                         CUtensorMapFloatOOBfill);
  static Fn enc = nullptr;
  if (!enc) {
    void* fp = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fp, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return -1;
    enc = reinterpret_cast<Fn>(fp);
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (bs % 8) || (ss % 8) || (hs % 8)) return -4;
  cuuint64_t dims[4] = {(cuuint64_t)a->hd, (cuuint64_t)a->S, (cuuint64_t)a->H, (cuuint64_t)a->B};
  cuuint64_t strides[3] = {(cuuint64_t)ss * 2, (cuuint64_t)(a->H > 1 ? hs : a->hd) * 2,
                           (cuuint64_t)(a->B > 1 ? bs : (long long)a->S * ss) * 2};
  cuuint32_t box[4] = {cols, rows, 1, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides,
                   box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1000 + (int)r;
}

static inline void fill_args(AttnArgs& p, const FtkAttnDesc* a) {
  p.B = a->B; p.H = a->H; p.S = a->S; p.causal = a->causal;
  p.scale = a->scale;
  p.sl2 = a->scale * 1.4426950408889634f;
  p.o = reinterpret_cast<const __nv_bfloat16*>(a->o);
  p.o_bs = a->o_bs; p.o_ss = a->o_ss; p.o_hs = a->o_hs;
  p.lse = a->lse; p.delta = a->delta;
  p.status = ftk_status_word();
}

static inline int device_sms() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!cache[dev]) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cache[dev] = n > 0 ? n : 148;
  }
  return cache[dev];
}

// Work items of `rows` rows each and the grid that walks them.
static inline int set_items(AttnArgs& p, const FtkAttnDesc* a, int rows, unsigned* grid) {
  const long long items = ((long long)a->S + rows - 1) / rows * a->H * a->B;
  if (items > 0x3fffffffll) return -2;
  p.n_tiles = (int)items;
  p.by_hb = FastDiv((uint32_t)(a->H * a->B));
  p.by_h = FastDiv((uint32_t)a->H);
  const int sms = device_sms();
  *grid = (unsigned)(items < sms ? items : sms);
  return 0;
}

template <typename K>
static inline int set_smem(K kernel, int bytes) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}


}  // namespace ftk
