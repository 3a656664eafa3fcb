// bf16 GEMM for sm_100a: TMA -> 128B-swizzled smem ring -> tcgen05.mma (fp32
// accumulators in TMEM, double buffered) -> tcgen05.ld epilogue.
//
//   D[l][M,N] = epi(alpha * A[l](M x K) * B[l](N x K)^T + bias[N]) (+ residual) (+ D)
//
// Both operands may be given K-major ("[rows, K]" row-major) or MN-major
// ("[K, rows]" row-major), so forward (x W^T), dgrad (dY W) and wgrad (dY^T x) of a
// Linear layer whose weight is [out, in] (reference: ft-kernel-cpu/src/lib.rs:17162
// linear_tensor_f64, :17226 linear_backward_f64) run without materialising a
// transpose.
//
// Determinism: within one launch K is reduced in ascending order by one CTA per output
// tile, so the result does not depend on the grid size.  Weight-gradient shapes (tiny
// output, very long K) use split-K: each split writes its fp32 partial tile to a
// workspace and a second kernel adds the partials in ascending split order - a fixed
// order again, so two runs give identical bits.
//
// One persistent CTA per SM, 10 warps: warp 0 issues TMA loads, warp 1 owns TMEM and
// issues the MMAs, warps 2..9 drain accumulators (warp w reads TMEM lane quarter w%4 and
// one half of the tile's columns).  Two accumulators let the epilogue of tile i overlap
// the mainloop of tile i+1.  The device code, including the collective-fused forms
// (all-gather -> GEMM, GEMM -> reduce-scatter), lives in gemm_kernel.cuh; this file holds
// the split-K reduction and the host launchers.
#include "gemm2_kernel.cuh"
#include "gemm_group_kernel.cuh"

#include <type_traits>

namespace ftk {

// D (+)= sum over splits (ascending) of ws[split]; 4 outputs per thread.
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ ws, void* __restrict__ D, long long M, long long N,
                     long long ldd, int splits, int out_fp32, int accumulate) {
  pdl_wait();
  pdl_trigger();
  const long long total4 = (M * N) >> 2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += stride) {
    // all partials of the element are requested before the first add (one memory latency, not `splits`);
    // the adds stay in ascending split order
    constexpr int U = 8;
    float4 t[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (k < splits) t[k] = __ldcg(reinterpret_cast<const float4*>(ws + (long long)k * M * N) + i);
    float4 s = t[0];
#pragma unroll
    for (int k = 1; k < U; ++k)
      if (k < splits) { s.x += t[k].x; s.y += t[k].y; s.z += t[k].z; s.w += t[k].w; }
    for (int k0 = U; k0 < splits; k0 += U) {
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (k0 + k < splits) t[k] = __ldcg(reinterpret_cast<const float4*>(ws + (long long)(k0 + k) * M * N) + i);
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (k0 + k < splits) { s.x += t[k].x; s.y += t[k].y; s.z += t[k].z; s.w += t[k].w; }
    }
    const long long e = i << 2;
    const long long r = e / N, c = e - r * N;
    if (out_fp32) {
      float* dp = reinterpret_cast<float*>(D) + r * ldd + c;
      if (accumulate) {
        const float4 o = *reinterpret_cast<float4*>(dp);
        s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
      }
      *reinterpret_cast<float4*>(dp) = s;
    } else {
      __nv_bfloat16* dp = reinterpret_cast<__nv_bfloat16*>(D) + r * ldd + c;
      if (accumulate) {
        const uint2 o = *reinterpret_cast<uint2*>(dp);
        const float2 a = unpack_bf16(o.x), b = unpack_bf16(o.y);
        s.x += a.x; s.y += a.y; s.z += b.x; s.w += b.y;
      }
      uint2 o;
      o.x = pack_bf16(s.x, s.y);
      o.y = pack_bf16(s.z, s.w);
      *reinterpret_cast<uint2*>(dp) = o;
    }
  }
}

__global__ void tick_i32_kernel(int* w) { *w += 1; }

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) !=
            cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 4-D bf16 tensor map {inner, outer, l0, l1} with 128B swizzle.
int ftk_make_tmap_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                       uint64_t l0, uint64_t l1, uint64_t ld_elems, uint64_t s0_elems,
                       uint64_t s1_elems, uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return -1;
  cuuint64_t dims[4] = {inner, outer, l0, l1};
  uint64_t st1 = ld_elems * 2;
  uint64_t st2 = (l0 > 1 ? s0_elems : outer * ld_elems) * 2;
  uint64_t st3 = (l1 > 1 ? s1_elems : (l0 > 1 ? s0_elems * l0 : outer * ld_elems)) * 2;
  if (st2 == 0) st2 = 16;
  if (st3 == 0) st3 = 16;
  cuuint64_t strides[3] = {st1, st2, st3};
  cuuint32_t box[4] = {box_inner, box_outer, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

static int num_sms() {
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

// cudaFuncSetAttribute applies to the current device only: remember per device what was set.
struct PerDeviceOnce {
  bool done[64] = {false};
  bool* slot() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    return &done[dev];
  }
};

// Divisors of the work-item decode for tiles of bm x bn.
static void set_divisors(GemmArgs& a, int bm, int bn) {
  const uint32_t tm = (uint32_t)((a.M + bm - 1) / bm), tn = (uint32_t)((a.N + bn - 1) / bn);
  a.by_tiles_m = FastDiv(tm);
  a.by_tiles_mn = FastDiv(tm * tn);
  a.by_batches = FastDiv((uint32_t)(a.L0 * a.L1));
  a.by_l0 = FastDiv((uint32_t)a.L0);
}

// m tiles per group of the pair kernel's walk.  With m fastest over all of them, the 74 tiles in flight hold up to 74 different
// row blocks of A against one or two column blocks of B, and an A that is larger than what L2 keeps is read again for every
// few columns: from memory, which costs time and, where the power limit sets the clock, the clock of the tensor pipe.  In
// groups, the tiles in flight are a patch of the output and A is read once (B again for each group, but from L2 if it fits).
// us, m fastest / groups of 4 / of 8, in bursts shorter than the power limit needs to act (in loops of 8 ms and more it lowers the
// clock until all walks are within 4 % of each other): 8192 x 2048 x 8192 194 / 187 / 188, 16384 x 4096 x 4096 403 / 343 / 347,
// 32768 x 8192 x 4096 1819 / 1523 / 1504, 65536 x 4096 x 1024 457 / 351 / 349; a weight gradient of a GPT-2 head, 50304 x 768 x 8192,
// 465 / 411 (groups of 4).  An A of up to half of L2 stays there as it is and B streams past it once: 4096 x 4096 x 4096 108 / 113 /
// 111 and 8192 x 50304 x 768, whose B is the larger operand, 535 / 585 / 549 (both in a loop).
// A B beyond L2 comes from memory once per group, so there are half as many, of 16: m fastest / groups of 8 / of 16
// 8192 x 50304 x 8192 5337 / 5587 / 5148, 8192 x 24576 x 8192 2515 / 2529 / 2376, 16384 x 32768 x 4096 3512 / 3322 / 2932,
// 16384 x 12288 x 8192 (192 MB) 2722 / 2548 / 2393.  With fewer than 32 row blocks three or more column blocks are in flight
// anyway, and a B of several times L2 is not worth reading again: 6144 x 50304 x 8192 3781 / 4064 / 3882, 6144 x 32768 x 8192
// 2405 / 2506 / 2447, 4096 x 24576 x 16384 2442 / 2553.
static uint32_t pair_group(long long M, long long N, long long K, uint32_t tm, uint32_t tn) {
  const long long a = 2 * M * K, b = 2 * N * K, MB = 1ll << 20;
  if (a <= 64 * MB || (tm < 32 && b > 320 * MB)) return tm;
  const uint32_t gm = b > 128 * MB ? 16 : (tn < 16 ? 4 : 8);
  return gm < tm ? gm : tm;
}

static void set_pair_groups(GemmArgs& a) {
  const uint32_t tm = a.by_tiles_m.d, tn = a.by_tiles_mn.d / tm;
  const uint32_t gm = pair_group(a.M, a.N, a.K, tm, tn), last = tm % gm ? tm % gm : gm;
  a.by_group = FastDiv(gm * tn);
  a.by_gm = FastDiv(gm);
  a.by_gm_last = FastDiv(last);
}

// The epilogue instantiation of a problem: a special kind where its parts are exactly those of the kind and every row is
// made of 16-byte segments, else the general one.
static int epilogue_kind(const GemmArgs& a) {
  const bool any_batch = a.L0 * a.L1 > 1;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (a.splits > 1)
    return (a.N % 4 == 0 && al(a.ws)) ? EPI_KIND_F32 : EPI_KIND_ANY;
  if (!al(a.D) || any_batch) return EPI_KIND_ANY;
  if (a.out_fp32)
    return (a.epi == FTK_EPI_NONE && !a.bias && !a.resid && !a.aux && a.ldd % 4 == 0 && a.N % 4 == 0) ? EPI_KIND_F32
                                                                                                    : EPI_KIND_ANY;
  if (a.accumulate || a.ldd % 8 || a.N % 8) return EPI_KIND_ANY;
  if (a.resid && (!al(a.resid) || a.ldr % 8)) return EPI_KIND_ANY;
  if (a.aux && !al(a.aux)) return EPI_KIND_ANY;
  if (a.epi == FTK_EPI_NONE && !a.aux) return a.resid ? EPI_KIND_RESID : EPI_KIND_PLAIN;
  if (a.epi == FTK_EPI_GELU_TANH && !a.resid) return a.aux ? EPI_KIND_GELU_AUX : EPI_KIND_GELU;
  if (a.epi == FTK_EPI_MUL_DGELU_TANH && a.resid && !a.aux && !a.bias) return EPI_KIND_DGELU;
  return EPI_KIND_ANY;
}

template <int BN, int KIND>
static int launch_gemm_kind(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmArgs a, int max_ctas,
                            cudaStream_t stream) {
  using Cfg = GemmCfg<BN>;
  static PerDeviceOnce once;
  bool* attr_set_p = once.slot();
  if (!*attr_set_p) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_sm100_kernel<BN, 0, KIND>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
    if (e != cudaSuccess) return (int)e;
    *attr_set_p = true;
  }
  set_divisors(a, G_BM, BN);
  long long items = (long long)((a.M + G_BM - 1) / G_BM) * ((a.N + BN - 1) / BN) * a.L0 * a.L1 * a.splits;
  if (items > 0x7fffffffll) return -2;
  int grid = (int)(items < max_ctas ? items : max_ctas);
  if (grid <= 0) return 0;
  CommArgs none;
  memset(&none, 0, sizeof(none));
  launch_pdl(gemm_bf16_sm100_kernel<BN, 0, KIND>, grid, G_THREADS, Cfg::SMEM, stream, tmA, tmB, tmA, a, none);
  return (int)cudaGetLastError();
}

// CTA-pair kernel: grid = 2 CTAs per cluster, at most sms / 2 clusters.
// Weight of the pair tiles in the tile-choice model: 1, the model's times are measured ones.  The environment variable
// FT_GEMM_PAIR_COST changes it to its value / 0.92 (0.92 is neutral; a large value rules the pair kernel out).
static double pair_cost_scale() {
  static double c = -1.0;
  if (c < 0.0) {
    const char* e = getenv("FT_GEMM_PAIR_COST");
    c = (e && atof(e) > 0.0) ? atof(e) / 0.92 : 1.0;
  }
  return c;
}
template <int BN, int KIND>
static int launch_gemm_pair_kind(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmArgs a, int max_ctas,
                                 cudaStream_t stream) {
  using Cfg = PairCfg<BN>;
  static PerDeviceOnce once;
  bool* attr_set_p = once.slot();
  if (!*attr_set_p) {
    cudaError_t e = cudaFuncSetAttribute(gemm2_bf16_sm100_kernel<BN, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg::SMEM);
    if (e != cudaSuccess) return (int)e;
    *attr_set_p = true;
  }
  set_divisors(a, 2 * G_BM, BN);
  set_pair_groups(a);
  const long long items = (long long)((a.M + 255) / 256) * ((a.N + BN - 1) / BN) * a.L0 * a.L1 * a.splits;
  if (items > 0x7fffffffll) return -2;
  long long pairs = max_ctas / 2;
  if (items < pairs) pairs = items;
  if (pairs <= 0) return 0;
  launch_pdl(gemm2_bf16_sm100_kernel<BN, KIND>, (unsigned)(2 * pairs), G_THREADS, Cfg::SMEM, stream, tmA, tmB, a);
  return (int)cudaGetLastError();
}

template <int BN, bool PAIR>
static int launch_gemm(int kind, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& a, int max_ctas,
                       cudaStream_t stream) {
  auto launch = [&](auto k) {
    if constexpr (PAIR)
      return launch_gemm_pair_kind<BN, decltype(k)::value>(tmA, tmB, a, max_ctas, stream);
    else
      return launch_gemm_kind<BN, decltype(k)::value>(tmA, tmB, a, max_ctas, stream);
  };
#define FT_LAUNCH_KIND(K) \
  case K: return launch(std::integral_constant<int, K>());
  switch (kind) {
    FT_LAUNCH_KIND(EPI_KIND_PLAIN)
    FT_LAUNCH_KIND(EPI_KIND_RESID)
    FT_LAUNCH_KIND(EPI_KIND_GELU)
    FT_LAUNCH_KIND(EPI_KIND_GELU_AUX)
    FT_LAUNCH_KIND(EPI_KIND_DGELU)
    FT_LAUNCH_KIND(EPI_KIND_F32)
    default: return launch(std::integral_constant<int, EPI_KIND_ANY>());
  }
#undef FT_LAUNCH_KIND
}

static int make_operand_maps(const FtkGemmDesc* g, int L0, int L1, int bn, CUtensorMap* tmA,
                             CUtensorMap* tmB) {
  int rc;
  if (!g->a_mn)
    rc = ftk_make_tmap_bf16(tmA, g->A, g->K, g->M, L0, L1, g->lda, g->a_s0, g->a_s1, G_BK, G_BM);
  else
    rc = ftk_make_tmap_bf16(tmA, g->A, g->M, g->K, L0, L1, g->lda, g->a_s0, g->a_s1, 64, G_BK);
  if (rc) return 1000 + rc;
  if (!g->b_mn)
    rc = ftk_make_tmap_bf16(tmB, g->B, g->K, g->N, L0, L1, g->ldb, g->b_s0, g->b_s1, G_BK, bn);
  else
    rc = ftk_make_tmap_bf16(tmB, g->B, g->N, g->K, L0, L1, g->ldb, g->b_s0, g->b_s1, 64, G_BK);
  if (rc) return 2000 + rc;
  return 0;
}

static void fill_gemm_args(GemmArgs& a, const FtkGemmDesc* g, int L0, int L1) {
  a.M = g->M; a.N = g->N; a.K = g->K; a.L0 = L0; a.L1 = L1;
  a.a_mn = g->a_mn ? 1 : 0; a.b_mn = g->b_mn ? 1 : 0;
  a.D = g->D; a.ldd = g->ldd; a.d_s0 = g->d_s0; a.d_s1 = g->d_s1;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(g->bias);
  a.resid = reinterpret_cast<const __nv_bfloat16*>(g->resid);
  a.ldr = g->ldr; a.r_s0 = g->r_s0; a.r_s1 = g->r_s1;
  a.aux = reinterpret_cast<__nv_bfloat16*>(g->aux);
  a.alpha = g->alpha; a.epi = g->epi; a.out_fp32 = g->out_fp32; a.accumulate = g->accumulate;
  a.splits = 1;
  a.ws = reinterpret_cast<float*>(g->workspace);
  a.status = ftk_status_word();
  a.seg_counts = g->seg_counts;
  a.seg_rows = g->seg_rows;
}

}  // namespace ftk

using namespace ftk;

// flags[0..n) = *epoch with system-scope release stores (the flags may live on another GPU); launched
// behind the copy whose arrival they announce, on the same stream.
__global__ void set_flags_sys_kernel(int* flags, int n, const int* __restrict__ epoch) {
  const int e = *epoch;
  __threadfence_system();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(flags + i), "r"(e) : "memory");
}
extern "C" int ftk_set_flags_sys(int* flags, int n, const int* epoch, void* stream_v) {
  if (!flags || !epoch || n <= 0) return -2;
  // one warp: it must find room on an SM beside a resident GEMM CTA (the consumer that waits for these flags)
  set_flags_sys_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(flags, n, epoch);
  return (int)cudaGetLastError();
}
// One device-to-device copy on a stream (local or peer destination): the copy engines move it, no SM is used.
extern "C" int ftk_copy_async(void* dst, const void* src, long long bytes, void* stream_v) {
  if (!dst || !src || bytes <= 0) return -2;
  return (int)cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDeviceToDevice,
                              reinterpret_cast<cudaStream_t>(stream_v));
}

extern "C" int ftk_tick_i32(int* word, void* stream_v) {
  if (!word) return -2;
  tick_i32_kernel<<<1, 1, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(word);
  return (int)cudaGetLastError();
}

// Argument checks and tile choice shared by the launcher and the plan query.  Returns 0 and
// (bn, splits), or a negative argument error.  bn > 256 stands for the CTA-pair kernel with 256 x (bn - 256) tiles.
static int plan_gemm(const FtkGemmDesc* g, int* bn_out, int* splits_out) {
  if (!g || g->M <= 0 || g->N <= 0 || g->K <= 0) return -2;
  const int L0 = g->L0 > 0 ? g->L0 : 1, L1 = g->L1 > 0 ? g->L1 : 1;
  // alignment rules of the tiled TMA copies: 16-byte base, 16-byte strides.
  if ((reinterpret_cast<uintptr_t>(g->A) & 15) || (reinterpret_cast<uintptr_t>(g->B) & 15)) return -3;
  if ((g->lda % 8) || (g->ldb % 8)) return -4;
  if ((L0 > 1 && ((g->a_s0 % 8) || (g->b_s0 % 8))) || (L1 > 1 && ((g->a_s1 % 8) || (g->b_s1 % 8))))
    return -4;

  const int sms = g->max_ctas > 0 ? g->max_ctas : num_sms();
  // Tile choice by modelled time: waves x (fixed cost of a tile + its k-blocks).  A k-block of 64 takes the tensor pipe
  // 2 BN cycles on one SM or on a pair; with every SM loading, operand delivery from L2 makes that longer by the
  // measured amounts below, in proportion to the SMs in use.  Measured against the model (us, 256 x 256 / 256 x 192 /
  // 256 x 128 pairs, then 128 x 256 / 192 / 128; all L2-resident): 8192 x 768 x 3072 36.7 / 31.3 / 34.5, 40.6 / 37.6 / 38.9;
  // 1500 x 1280 x 5120 29.6 / 23.7 / 19.3, 29.2 / 23.4 / 21.6; 1500 x 3840 x 1280 17.8 / 14.7 / 16.0, 18.6 / 15.5 / 17.9;
  // 8192 x 2304 x 768 21.9 / 23.0 / 25.0, 24.4 / 26.6 / 27.7.  224 and 160 columns (pairs only): 8192 x 2304 x 768 23.3 / 23.8,
  // 1500 x 1280 x 5120 26.7 / 21.7 beside 29.8 / 25.4 / 20.1, 512 x 8192 x 8192 46.9 / 63.4 beside 50.1 / 67.0 / 55.6.
  // Split-K (weight-gradient shapes: few output tiles, long reduction) is considered when the
  // epilogue is a plain store and the caller supplied a workspace.
  const int kblocks = (g->K + G_BK - 1) / G_BK;
  if (g->seg_counts && g->seg_rows <= 0) return -2;
  const bool splittable = g->epi == FTK_EPI_NONE && !g->bias && !g->resid && !g->aux && g->workspace &&
                          (g->N % 4 == 0) && (g->ldd % 4 == 0) && L0 * L1 == 1 && !g->seg_counts;
  // A split costs the reduction kernel: s fp32 partials read, the output written (and read when
  // it accumulates) at ~4 TB/s plus a launch - 17 us for an [8192, 768] bf16 output with two splits, which is
  // why an activation-sized output is hardly ever worth splitting while a weight gradient is.
  auto split_penalty = [&](int s) {
    if (s <= 1) return 0.0;
    const double mn = (double)g->M * (double)g->N;
    const double bytes = mn * 4.0 * s + mn * (g->out_fp32 ? 4.0 : 2.0) * (g->accumulate ? 2.0 : 1.0);
    return bytes / 4.0e6 + 3.0;
  };
  // An operand whose rows are not whole 128-byte lines: every 128-byte row of a box straddles two lines, which the wide pair
  // tiles, with the fewest rows per MMA, feel least.  us per k-block with no, one and both operands off: 1500 x 1000 x 5000, B
  // [K, N], on 256 x 128 pairs 0.22 / 0.28 / 0.38; 8192 x 768 x 3000 on 256 x 256 pairs 0.33 and 0.43 with both, on 128 x 192
  // 0.31 and 0.58; weight gradients of 2048 x 640 and 2136 x 632 on 256 x 128 pairs 0.20 and 0.36.
  const int off_lines = (g->lda % 64 != 0 ? 1 : 0) + (g->ldb % 64 != 0 ? 1 : 0);
  auto cost = [&](int bn, int s) {
    const bool pair = bn > 256;
    const int w = pair ? bn - 256 : bn;
    // 256, 224, 192, 160, 128 columns
    const int wi = (256 - w) / 32;
    static const double tile_us[5] = {0.4, 0.3, 0.1, 0.2, 0.3}, mma_us[5] = {0.278, 0.244, 0.21, 0.176, 0.143};
    static const double pair_us[5] = {0.375, 0.35, 0.32, 0.30, 0.235}, one_us[5] = {0.42, 0.0, 0.385, 0.0, 0.27};
    static const double exposed_us[5] = {0.75, 0.7, 0.55, 0.3, 0.0};
    const double tile = tile_us[wi], mma = mma_us[wi], full = pair ? pair_us[wi] : one_us[wi];
    const long long items = ((g->M + (pair ? 255 : 127)) / (pair ? 256 : 128)) * (long long)((g->N + w - 1) / w) * L0 * L1 * s;
    const long long units = pair ? sms / 2 : sms;
    const long long waves = (items + units - 1) / units;
    const double busy = items < units ? (double)items / (double)units : 1.0;
    // the last tile's epilogue and a pair's hand-shakes are not hidden: 128 x 192 x 64 takes 4.1 / 4.7 / 4.8 us on one
    // SM and 4.6 / 5.1 / 5.3 us on a pair
    const double off = bn > 256 ? (w == 256 ? 1.2 : 1.3) : 1.35, lines = off_lines == 0 ? 1.0 : (off_lines == 1 ? off : off * off);
    const double exposed = exposed_us[wi] + (pair ? 0.5 : 0.0);
    return ((double)waves * (tile + (double)kblocks / s * (mma + (full - mma) * busy) * lines) + exposed) *
               (pair ? pair_cost_scale() : 1.0) + split_penalty(s);
  };
  auto split_ok = [&](int s) {
    if (s == 1) return true;
    if (!splittable || g->split_k == 1 || kblocks / s < 8) return false;
    return (long long)s * g->M * g->N * 4 <= g->workspace_bytes;
  };
  static const int bn_opts[8] = {512, 480, 448, 416, 384, 256, 192, 128};
  static const int s_opts[8] = {1, 2, 3, 4, 6, 8, 12, 16};
  int bn = g->force_bn, splits = 1;
  double best = 1e30;
  for (int bi = 0; bi < 8; ++bi) {
    if (bn_opts[bi] > 256 && (sms < 2 || g->M < 256 || g->seg_counts)) continue;
    if (g->force_bn && bn_opts[bi] != g->force_bn) continue;
    // 160 and 224 columns fill the last wave of forward products: with bias, in a captured loop with the operands in L2, 1500 x 3840 x
    // 1280 in 144 tiles of 160 12.6 us, 120 of 192 13.5; 1500 x 5120 x 1280 in 138 of 224 15.2, 120 of 256 16.6.  A half of 80 or 112
    // columns of a B given [K, N] loads 128 all the same, and nothing is gained: in a sequence of calls 17.2 and 17.5, 21.7 and 20.5.
    if ((bn_opts[bi] == 416 || bn_opts[bi] == 480) && g->b_mn && !g->force_bn) continue;
    for (int si = 0; si < 8; ++si) {
      const int s = s_opts[si];
      if (g->split_k > 1 && s != g->split_k && s != 1) continue;
      if (!split_ok(s)) continue;
      const double c = cost(bn_opts[bi], s);
      if (c < best - 1e-9) {
        best = c;
        bn = bn_opts[bi];
        splits = s;
      }
    }
  }
  if (g->split_k > 1 && split_ok(g->split_k)) splits = g->split_k;
  if (bn != 128 && bn != 192 && bn != 256 && bn != 384 && bn != 416 && bn != 448 && bn != 480 && bn != 512) return -5;
  // a forced pair tile needs two CTAs (without them nothing would run), and pair tiles know no rows that are not in use
  if (bn > 256 && (sms < 2 || g->seg_counts)) return -5;
  *bn_out = bn;
  *splits_out = splits;
  return 0;
}

template <int BN, int KIND>
static int launch_group(const GroupMaps& maps, const GroupArgs& ga, int pairs, cudaStream_t stream) {
  constexpr int SMEM = PairCfg<BN>::SMEM;
  static PerDeviceOnce once;
  bool* attr_set_p = once.slot();
  if (!*attr_set_p) {
    cudaError_t e = cudaFuncSetAttribute(gemm_group_bf16_sm100_kernel<BN, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SMEM);
    if (e != cudaSuccess) return (int)e;
    *attr_set_p = true;
  }
  launch_pdl(gemm_group_bf16_sm100_kernel<BN, KIND>, 2 * pairs, G_THREADS, SMEM, stream, maps, ga);
  return (int)cudaGetLastError();
}

// Tile width of a grouped launch, its tiles and its CTAs: whole pairs, or one CTA where no pair is allowed.
struct GroupPlan {
  int bn, total, ctas;
};
// The wide tile loads 40 KB per CTA for the work that two 256 x 192 tiles load 64 KB for (an MN-major half of 96 columns comes in
// two boxes of 64), but has one accumulator, so its epilogue is not hidden.  Modelled time: waves x (fixed + k-blocks), in us:
// 1.2 + 0.34 per k-block of 64 and 4.5 + 0.62.  Measured, 192 / 384 columns, back to back without and with the power limit: the
// four weight gradients of a block of 768 over 8192 rows 88.8 / 82.1 and 111.1 / 97.5, over 2048 rows 28.7 / 28.8, over 512 rows
// 13.4 / 14.3; of a block of 1024 over 8192 rows 168.9 / 158.6 and 203.5 / 186.7, of 512 over 4096 rows (70 and 44 tiles, one wave
// both) 25.8 / 41.2; an MLP of 2048 over 8192 rows 449 / 409 and 578 / 491; a block of 1280 over 4096 rows (6 and 4 waves)
// 134 / 155.
static GroupPlan plan_group(const FtkGemmDesc* descs, int n) {
  const int sms = descs[0].max_ctas > 0 ? descs[0].max_ctas : num_sms();
  const double kblocks = (double)((descs[0].K + G_BK - 1) / G_BK);
  GroupPlan best = {GG_BN, 0, 1};
  double best_us = 1e30;
  for (int bn : {GG_BN, GG_BN_WIDE}) {
    long long total = 0;
    for (int p = 0; p < n; ++p)
      total += (long long)((descs[p].M + 2 * G_BM - 1) / (2 * G_BM)) * ((descs[p].N + bn - 1) / bn);
    const long long units = sms > 1 ? sms / 2 : 1, waves = (total + units - 1) / units;
    const double us = waves * (bn == GG_BN ? 1.2 + 0.34 * kblocks : 4.5 + 0.62 * kblocks);
    if (us < best_us) {
      best_us = us;
      best.bn = bn;
      best.total = (int)total;
    }
  }
  const int pairs = best.total < sms / 2 ? best.total : sms / 2;
  best.ctas = pairs > 0 ? 2 * pairs : 1;
  return best;
}

// Grouped launch: `n` (1..8) independent products with the same K and operand layouts, fp32 outputs with a plain
// store or accumulate epilogue, in one persistent kernel of pair tiles (see gemm_group_kernel.cuh).
extern "C" int ftk_gemm_group_bf16(const FtkGemmDesc* descs, int n, void* stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (!descs || n < 1 || n > GG_MAX) return -2;
  GroupArgs ga = {};
  GroupMaps maps;
  memset(&maps, 0, sizeof(maps));
  const FtkGemmDesc& g0 = descs[0];
  ga.n = n; ga.K = g0.K; ga.a_mn = g0.a_mn ? 1 : 0; ga.b_mn = g0.b_mn ? 1 : 0; ga.alpha = g0.alpha;
  ga.status = ftk_status_word();
  if (!ga.status) return -6;
  for (int p = 0; p < n; ++p)
    if (descs[p].M <= 0 || descs[p].N <= 0) return -2;
  const GroupPlan plan = plan_group(descs, n);
  const int bn = plan.bn;
  int total = 0;
  for (int p = 0; p < n; ++p) {
    const FtkGemmDesc* g = &descs[p];
    if (g->M <= 0 || g->N <= 0 || g->K != g0.K || (g->a_mn ? 1 : 0) != ga.a_mn || (g->b_mn ? 1 : 0) != ga.b_mn ||
        g->alpha != g0.alpha)
      return -2;
    if ((g->L0 > 1) || (g->L1 > 1) || !g->out_fp32 || g->epi != FTK_EPI_NONE || g->bias || g->resid || g->aux ||
        g->seg_counts || !g->D)
      return -7;
    if ((reinterpret_cast<uintptr_t>(g->A) & 15) || (reinterpret_cast<uintptr_t>(g->B) & 15)) return -3;
    if ((g->lda % 8) || (g->ldb % 8)) return -4;
    int rc = make_operand_maps(g, 1, 1, bn / 2, &maps.a[p], &maps.b[p]);
    if (rc) return rc;
    ga.M[p] = g->M; ga.N[p] = g->N;
    ga.D[p] = reinterpret_cast<float*>(g->D);
    ga.ldd[p] = g->ldd;
    ga.accumulate[p] = g->accumulate ? 1 : 0;
    ga.by_tiles_m[p] = FastDiv((uint32_t)((g->M + 2 * G_BM - 1) / (2 * G_BM)));
    total += ((g->M + 2 * G_BM - 1) / (2 * G_BM)) * ((g->N + bn - 1) / bn);
    ga.tile_end[p] = total;
  }
  for (int p = n; p < GG_MAX; ++p) ga.tile_end[p] = total;
  if (plan.ctas < 2) {
    // one CTA is all the caller allows: the products in turn, same k order, so the same bits
    for (int p = 0; p < n; ++p) {
      FtkGemmDesc one = descs[p];
      one.force_bn = GG_BN;
      one.split_k = 1;
      one.max_ctas = 1;
      const int rc = ftk_gemm_bf16(&one, stream_v);
      if (rc) return rc;
    }
    return 0;
  }
  bool aligned = true;
  for (int p = 0; p < n; ++p)
    aligned = aligned && ga.N[p] % 4 == 0 && ga.ldd[p] % 4 == 0 && (reinterpret_cast<uintptr_t>(ga.D[p]) & 15) == 0;
  const int pairs = plan.ctas / 2;
  if (bn == GG_BN_WIDE)
    return aligned ? launch_group<GG_BN_WIDE, EPI_KIND_F32>(maps, ga, pairs, stream)
                   : launch_group<GG_BN_WIDE, EPI_KIND_ANY>(maps, ga, pairs, stream);
  return aligned ? launch_group<GG_BN, EPI_KIND_F32>(maps, ga, pairs, stream)
                 : launch_group<GG_BN, EPI_KIND_ANY>(maps, ga, pairs, stream);
}

// CTAs that the grouped launch takes: never more than max_ctas.  Launches nothing.
extern "C" int ftk_gemm_group_ctas(const FtkGemmDesc* descs, int n) {
  if (!descs || n < 1 || n > GG_MAX) return -2;
  return plan_group(descs, n).ctas;
}

// Columns of its tiles: 192 or 384, or 0 where one CTA is all that max_ctas allows and the products run in turn.  Launches nothing.
extern "C" int ftk_gemm_group_width(const FtkGemmDesc* descs, int n) {
  if (!descs || n < 1 || n > GG_MAX) return -2;
  const GroupPlan plan = plan_group(descs, n);
  return plan.ctas < 2 ? 0 : plan.bn;
}

// Which kernel ftk_gemm_bf16 would launch for this problem: *bn = 128 / 192 / 256 (single-CTA tile 128 x bn) or
// 384 to 512 in steps of 32 (CTA-pair kernel, tiles of 256 x (bn - 256)); *splits = split-K factor.  Launches nothing.
extern "C" int ftk_gemm_plan(const FtkGemmDesc* g, int* bn, int* splits) {
  if (!bn || !splits) return -2;
  return plan_gemm(g, bn, splits);
}

// Row blocks of 256 that the pair kernel would walk as one group for this problem (all of them: m fastest), 0 for a single-CTA
// tile.  Launches nothing.
extern "C" int ftk_gemm_walk(const FtkGemmDesc* g) {
  int bn = 0, splits = 1;
  const int rc = plan_gemm(g, &bn, &splits);
  if (rc || bn <= 256) return rc;
  return (int)pair_group(g->M, g->N, g->K, (uint32_t)((g->M + 255) / 256), (uint32_t)((g->N + bn - 257) / (bn - 256)));
}

// (one event per device and thread, re-recorded per call: another thread's record between this one's record and wait would
// order the second stream behind the wrong work)
extern "C" int ftk_stream_order(void* first, void* then) {
  static thread_local cudaEvent_t ev[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!ev[dev]) {
    cudaError_t e = cudaEventCreateWithFlags(&ev[dev], cudaEventDisableTiming);
    if (e != cudaSuccess) return (int)e;
  }
  cudaError_t e = cudaEventRecord(ev[dev], reinterpret_cast<cudaStream_t>(first));
  if (e == cudaSuccess) e = cudaStreamWaitEvent(reinterpret_cast<cudaStream_t>(then), ev[dev], 0);
  return (int)e;
}

extern "C" int ftk_gemm_bf16(const FtkGemmDesc* g, void* stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  int bn = 0, splits = 1;
  int prc = plan_gemm(g, &bn, &splits);
  if (prc) return prc;
  const int L0 = g->L0 > 0 ? g->L0 : 1, L1 = g->L1 > 0 ? g->L1 : 1;
  const int sms = g->max_ctas > 0 ? g->max_ctas : num_sms();

  CUtensorMap tmA, tmB;
  int rc = make_operand_maps(g, L0, L1, bn > 256 ? (bn - 256) / 2 : bn, &tmA, &tmB);   // a pair stages half of B per CTA
  if (rc) return rc;

  GemmArgs a;
  fill_gemm_args(a, g, L0, L1);
  a.splits = splits;
  if (!a.status) return -6;
  if (a.accumulate && !a.out_fp32 && !a.resid && splits == 1 && a.epi < FTK_EPI_MUL_DGELU_TANH) {
    // A bf16 output that is added to is its own residual: the same sum, rounded once, and the staged epilogue instead of the
    // general one (8192 x 768 x 3072 112 -> 29 us).  Every element is read by the warp that then writes it.
    a.resid = reinterpret_cast<const __nv_bfloat16*>(a.D);
    a.ldr = a.ldd;
    a.r_s0 = a.d_s0;
    a.r_s1 = a.d_s1;
    a.accumulate = 0;
  }
  const int kind = epilogue_kind(a);
  rc = bn == 512   ? launch_gemm<256, true>(kind, tmA, tmB, a, sms, stream)
       : bn == 480 ? launch_gemm<224, true>(kind, tmA, tmB, a, sms, stream)
       : bn == 448 ? launch_gemm<192, true>(kind, tmA, tmB, a, sms, stream)
       : bn == 416 ? launch_gemm<160, true>(kind, tmA, tmB, a, sms, stream)
       : bn == 384 ? launch_gemm<128, true>(kind, tmA, tmB, a, sms, stream)
       : bn == 256 ? launch_gemm<256, false>(kind, tmA, tmB, a, sms, stream)
       : bn == 192 ? launch_gemm<192, false>(kind, tmA, tmB, a, sms, stream)
                   : launch_gemm<128, false>(kind, tmA, tmB, a, sms, stream);
  if (rc || splits == 1) return rc;
  const long long total4 = ((long long)g->M * g->N) >> 2;
  long long blocks = (total4 + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  cudaStream_t rs = g->reduce_stream ? reinterpret_cast<cudaStream_t>(g->reduce_stream) : stream;
  if (rs != stream) {
    const int erc = ftk_stream_order(stream, rs);      // reduction on its own stream, ordered behind the GEMM
    if (erc) return erc;
  }
  launch_pdl(splitk_reduce_kernel, (unsigned)blocks, 256, 0, rs, a.ws, g->D, g->M, g->N, g->ldd, splits,
                                                         g->out_fp32, g->accumulate);
  return (int)cudaGetLastError();
}

// GEMM fused with all-gather of an operand or reduce-scatter of the output (see ftk_api.h).
extern "C" int ftk_gemm_comm_bf16(const FtkGemmDesc* g, const FtkCommDesc* cd, void* stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (!g || !cd || g->M <= 0 || g->N <= 0 || g->K <= 0) return -2;
  if (cd->world < 1 || cd->world > FTK_MAX_RANKS || cd->rank < 0 || cd->rank >= cd->world) return -2;
  if (cd->mode < FTK_COMM_GATHER_A || cd->mode > FTK_COMM_SCATTER_D || !cd->epoch) return -2;
  if ((g->L0 > 1) || (g->L1 > 1)) return -2;
  if ((reinterpret_cast<uintptr_t>(g->A) & 15) || (reinterpret_cast<uintptr_t>(g->B) & 15)) return -3;
  if ((g->lda % 8) || (g->ldb % 8)) return -4;
  if (cd->chunk_rows <= 0 || cd->chunk_rows % G_BM) return -7;
  constexpr int BN = 256;
  const long long rows_total = (long long)cd->chunk_rows * cd->world;

  CommArgs c;
  memset(&c, 0, sizeof(c));
  c.mode = cd->mode; c.rank = cd->rank; c.world = cd->world; c.chunk_rows = cd->chunk_rows;
  c.epoch = cd->epoch;
  const int sms = g->max_ctas > 0 ? g->max_ctas : num_sms();
  // gathers: CTAs that only move data (default 20); reduce-scatter: every CTA reduces after its
  // GEMM tiles, dedicated CTAs are optional (default none)
  c.comm_ctas = cd->comm_ctas > 0 ? cd->comm_ctas : (cd->mode == FTK_COMM_SCATTER_D ? 0 : 20);
  if (cd->mode != FTK_COMM_SCATTER_D && (cd->push == 2 || cd->push == 3)) {
    c.comm_ctas = 0;    // 2: the shards arrive by copy engine; 3: the epilogue warps of every CTA push them
  } else if (cd->comm_ctas <= 0 && cd->mode != FTK_COMM_SCATTER_D && cd->push) {
    c.comm_ctas = 16;
  } else if (cd->comm_ctas <= 0 && cd->mode != FTK_COMM_SCATTER_D) {
    // Split the SMs between copying and computing in proportion to the work: a copy CTA keeps
    // 128 KB of peer loads in flight, which at NVLink latency under load is ~13 GB/s (measured
    // at 2 and 8 ranks), a compute CTA delivers its share of the sustained GEMM rate.
    const bool bk = cd->mode == FTK_COMM_GATHER_B && g->b_mn;
    const double row_bytes = 2.0 * (double)(bk ? g->N : g->K);
    const double remote = (double)(cd->world - 1) * (double)cd->chunk_rows * row_bytes;
    const double comm_work = remote / 13e9;
    const double gemm_work = 2.0 * (double)g->M * (double)g->N * (double)g->K / (1.4e15 / (double)sms);
    int cc = (int)(sms * comm_work / (comm_work + gemm_work) + 0.5);
    if (cc < 12) cc = 12;
    if (cc > 64) cc = 64;
    if (cd->world == 1) cc = 32;   // nothing to fetch: the copy CTAs only stage the own chunk
    c.comm_ctas = cc;
  }
  if (c.comm_ctas >= sms) return -7;

  if (cd->mode == FTK_COMM_SCATTER_D) {
    if (rows_total != g->M || (g->N % 8) || (g->ldd % 8) || (g->resid && (g->ldr % 8))) return -7;
    if (g->epi != FTK_EPI_NONE || g->aux) return -7;
    for (int r = 0; r < cd->world; ++r) {
      if (!cd->inbox[r] || !cd->arrive[r]) return -2;
      c.inbox[r] = reinterpret_cast<__nv_bfloat16*>(cd->inbox[r]);
      c.arrive[r] = cd->arrive[r];
    }
  } else {
    const bool ga = cd->mode == FTK_COMM_GATHER_A;
    // the staged operand must be contiguous [rows, K] so that a subtile is one byte range
    // (B given MN-major, i.e. [K, N] row-major, is sharded along K: dgrad with a sharded weight)
    const bool bk = !ga && g->b_mn;
    if (ga ? (g->a_mn || g->lda != g->K || rows_total != g->M)
           : (bk ? (g->ldb != g->N || rows_total != g->K) : (g->ldb != g->K || rows_total != g->N)))
      return -7;
    c.sub_bytes = (long long)G_BM * (bk ? g->N : g->K) * 2;
    if (c.sub_bytes > G_COPY_SLOT ? (c.sub_bytes % G_COPY_SLOT) : (c.sub_bytes % 16)) return -7;
    if (!cd->sub_flags) return -2;
    c.full = reinterpret_cast<uint8_t*>(const_cast<void*>(ga ? g->A : g->B));
    c.sub_flags = cd->sub_flags;
    c.ready_local = cd->push ? nullptr : cd->ready_local;
    c.push = cd->push == 3 ? 3 : (cd->push ? 1 : 0);
    for (int r = 0; r < cd->world; ++r) {
      if (cd->push) {
        // only the own shard is read; peers' staging buffers and flag arrays are written
        if (!cd->full_peer[r] || !cd->flags_peer[r] || (reinterpret_cast<uintptr_t>(cd->full_peer[r]) & 15)) return -2;
        c.full_peer[r] = reinterpret_cast<uint8_t*>(cd->full_peer[r]);
        c.flags_peer[r] = cd->flags_peer[r];
        if (r != cd->rank) continue;
      }
      if (!cd->src[r] || (reinterpret_cast<uintptr_t>(cd->src[r]) & 15)) return -3;
      c.src[r] = reinterpret_cast<const uint8_t*>(cd->src[r]);
      c.ready_peer[r] = cd->ready_peer[r];
      if (!cd->push && cd->ready_local && r != cd->rank && !cd->ready_peer[r]) return -2;
    }
    if (cd->push && (c.full_peer[cd->rank] != c.full || c.flags_peer[cd->rank] != c.sub_flags)) return -2;
  }

  CUtensorMap tmA, tmB;
  int rc = make_operand_maps(g, 1, 1, BN, &tmA, &tmB);
  if (rc) return rc;
  GemmArgs a;
  fill_gemm_args(a, g, 1, 1);
  if (!a.status) return -6;

  using Cfg = GemmCfg<BN>;
  constexpr int COMM_SMEM = Cfg::SMEM;
  static PerDeviceOnce once;
  bool* attr_set_p = once.slot();
  if (!*attr_set_p) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_sm100_kernel<BN, 1, EPI_KIND_ANY>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, COMM_SMEM);
    if (e != cudaSuccess) return (int)e;
    *attr_set_p = true;
  }
  set_divisors(a, G_BM, BN);
  const long long items = (long long)((a.M + G_BM - 1) / G_BM) * ((a.N + BN - 1) / BN);
  long long n_compute = sms - c.comm_ctas;
  if (items < n_compute) n_compute = items;
  const int grid = (int)n_compute + c.comm_ctas;   // all CTAs resident: one per SM
  // tiles inside this rank's own shard are read from the shard, not from the staging buffer
  CUtensorMap tmOwn = tmA;
  if (cd->mode == FTK_COMM_GATHER_A)
    rc = ftk_make_tmap_bf16(&tmOwn, cd->src[cd->rank], g->K, cd->chunk_rows, 1, 1, g->K, 0, 0, G_BK, G_BM);
  else if (cd->mode == FTK_COMM_GATHER_B && !g->b_mn && cd->chunk_rows >= BN)
    rc = ftk_make_tmap_bf16(&tmOwn, cd->src[cd->rank], g->K, cd->chunk_rows, 1, 1, g->K, 0, 0, G_BK, BN);
  if (rc) return 3000 + rc;
  gemm_bf16_sm100_kernel<BN, 1, EPI_KIND_ANY><<<grid, G_THREADS, COMM_SMEM, stream>>>(tmA, tmB, tmOwn, a, c);
  return (int)cudaGetLastError();
}
