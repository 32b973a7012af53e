// C entry points of the tcgen05 GEMM (see gemm_tcgen05.cuh for the kernel).
#include <cstdlib>

#include "../common/host_utils.h"
#include "gemm_tcgen05.cuh"
#include "gemm_2cta.cuh"
#include "gemm_few_rows.cuh"
#include "ofb_kernels.h"

namespace ofb {

// Whether shapes that fill the machine use the two-SM kernel unless told otherwise.
constexpr bool kDefault2Cta = true;
// Up to 64 rows the product is a stream of weights (gemm_few_rows.cuh). With 33 rows and more, whose tiles every CTA reads besides, only
// while the 128-column tiles fit the machine at once: 64 x 32768 x 2048 33.7 against 40.7 us with the tiled kernels, 64 x 40960 x 2048
// 51.4 against 43.9, 33 x 40960 x 2048 45.4 against 42.3 (17 x 50304 x 2048 44.7 against 60.4).
static bool few_rows(const OfbGemmArgs* a) { return a->M <= 32 || (a->M <= 64 && a->N <= 32768); }

template <int BN, int A_MN, int B_MN, int ST, int MINB, int EPI>
static int launch_gemm_as(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmShape& shp, const GemmEpilogue& ep,
                       int* status, int max_ctas, cudaStream_t stream) {
  using Cfg = GemmCfg<BN, ST>;
  auto kern = gemm_bf16_tcgen05_kernel<BN, A_MN, B_MN, ST, MINB, EPI>;
  OFB_CUDA_OK_ONCE_PER_DEVICE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    OFB_CUDA_OK(cudaGetDevice(&dev));
    OFB_CUDA_OK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  const int tiles = ((shp.M + 127) / 128) * ((shp.N + BN - 1) / BN) * (shp.splits > 1 ? shp.splits : 1);
  int grid = tiles < sm_count * MINB ? tiles : sm_count * MINB;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  kern<<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(tmA, tmB, shp, ep, status);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

// The epilogue compiled for itself where there is one: activations of forward products (both operands K-major), gradients of
// activations in data gradients (B MN-major), fp32 results of weight gradients (A MN-major).
#define OFB_GEMM_BY_EPILOGUE(launch, ...)                                                                                          \
  switch (gemm_epilogue_kind(ep)) {                                                                                                \
    case kEpiLinear: return launch<__VA_ARGS__, kEpiLinear>(tmA, tmB, shp, ep, status, max_ctas, stream);                           \
    case kEpiGelu: if constexpr (!A_MN && !B_MN) return launch<__VA_ARGS__, kEpiGelu>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    case kEpiRelu: if constexpr (!A_MN && !B_MN) return launch<__VA_ARGS__, kEpiRelu>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    case kEpiGeluGrad: if constexpr (!A_MN && B_MN) return launch<__VA_ARGS__, kEpiGeluGrad>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    case kEpiReluGrad: if constexpr (!A_MN && B_MN) return launch<__VA_ARGS__, kEpiReluGrad>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    case kEpiMasked: if constexpr (!A_MN && B_MN) return launch<__VA_ARGS__, kEpiMasked>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    case kEpiWide: if constexpr (A_MN && B_MN) return launch<__VA_ARGS__, kEpiWide>(tmA, tmB, shp, ep, status, max_ctas, stream); break; \
    default: break;                                                                                                                \
  }                                                                                                                                \
  return launch<__VA_ARGS__, kEpiAny>(tmA, tmB, shp, ep, status, max_ctas, stream)

template <int BN, int A_MN, int B_MN, int ST = 0, int MINB = 1>
static int launch_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmShape& shp, const GemmEpilogue& ep,
                       int* status, int max_ctas, cudaStream_t stream) {
  OFB_GEMM_BY_EPILOGUE(launch_gemm_as, BN, A_MN, B_MN, ST, MINB);
}

template <int A_MN, int B_MN, int EPI>
static int launch_gemm_2cta_as(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmShape& shp, const GemmEpilogue& ep,
                            int* status, int max_ctas, cudaStream_t stream) {
  auto kern = gemm_bf16_2cta_kernel<A_MN, B_MN, EPI>;
  OFB_CUDA_OK_ONCE_PER_DEVICE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Gemm2Cfg::SMEM8_BYTES));
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    OFB_CUDA_OK(cudaGetDevice(&dev));
    OFB_CUDA_OK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  const int tiles = ((shp.M + 255) / 256) * ((shp.N + 255) / 256);
  int grid = 2 * tiles < sm_count ? 2 * tiles : (sm_count & ~1);
  if (max_ctas > 1 && grid > (max_ctas & ~1)) grid = max_ctas & ~1;
  kern<<<grid, Gemm2Cfg::THREADS, Gemm2Cfg::SMEM8_BYTES, stream>>>(tmA, tmB, shp, ep, status);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int A_MN, int B_MN>
static int launch_gemm_2cta(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmShape& shp, const GemmEpilogue& ep,
                            int* status, int max_ctas, cudaStream_t stream) {
  OFB_GEMM_BY_EPILOGUE(launch_gemm_2cta_as, A_MN, B_MN);
}
#undef OFB_GEMM_BY_EPILOGUE

template <int NP, int W_MN>
static int launch_gemm_few_rows(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmShape& shp, const GemmEpilogue& ep, int* status,
                                cudaStream_t stream) {
  using Cfg = FewRowsCfg<NP>;
  auto kern = gemm_few_rows_kernel<NP, W_MN>;
  OFB_CUDA_OK_ONCE_PER_DEVICE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(static_cast<unsigned>((shp.N + Cfg::BM - 1) / Cfg::BM * shp.splits));
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(shp.splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  OFB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, shp, ep, status));
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

// The K range of a tile is shared by CTAs (a cluster) as far as 256 of them hold the tiles at once (clusters do not fill all 296 places:
// 8 x 6144 x 2048, 48 tiles: five CTAs each 9.8 us, six 14.9) and each keeps four K blocks, with long K sixteen (8 x 3072 x 1024: four CTAs
// 6.7 us, eight 7.9; 8 x 4096 x 4096: four 11.0, eight 11.5; 8 x 4096 x 16384: four 30.1, eight 27.9).
static int gemm_few_rows(const OfbGemmArgs* a, const GemmEpilogue& ep, cudaStream_t stream) {
  const int tiles = (a->N + 127) / 128, kblocks = (a->K + 63) / 64;
  int parts = kblocks / 16 > 4 ? kblocks / 16 : kblocks / 4 < 4 ? kblocks / 4 : 4;
  if (parts > 8) parts = 8;
  if (parts > 256 / tiles) parts = 256 / tiles;
  if (parts < 1) parts = 1;
  const int kb_per = (kblocks + parts - 1) / parts;
  parts = (kblocks + kb_per - 1) / kb_per;          // no part without a K block
  const int np = a->M <= 16 ? 16 : a->M <= 32 ? 32 : 64;
  CUtensorMap tmW, tmX;
  if (!a->b_mn_major) {
    if (get_tensor_map(&tmW, a->B, 2, 2, a->K, a->N, 0, (uint64_t)a->ldb * 2, 0, 64, 128, 0, 3)) return -1;
  } else {
    if (get_tensor_map(&tmW, a->B, 2, 2, a->N, a->K, 0, (uint64_t)a->ldb * 2, 0, 64, 64, 0, 3)) return -1;
  }
  if (get_tensor_map(&tmX, a->A, 2, 2, a->K, a->M, 0, (uint64_t)a->lda * 2, 0, 64, np, 0, 3)) return -1;
  const GemmShape shp{a->M, a->N, a->K, parts};
  int* status = device_status_ptr();
#define OFB_FEW_ROWS(NP_)   if (np == NP_) return a->b_mn_major ? launch_gemm_few_rows<NP_, 1>(tmW, tmX, shp, ep, status, stream) : launch_gemm_few_rows<NP_, 0>(tmW, tmX, shp, ep, status, stream);
  OFB_FEW_ROWS(16)
  OFB_FEW_ROWS(32)
  OFB_FEW_ROWS(64)
#undef OFB_FEW_ROWS
  return fail("gemm: few rows");
}

static int gemm_mode_2cta() {
  // OFB_GEMM_2CTA=0 turns the two-SM kernel off, =1 forces it for every shape it supports.
  static int mode = -2;
  if (mode == -2) {
    const char* e = std::getenv("OFB_GEMM_2CTA");
    mode = e ? std::atoi(e) : -1;
  }
  return mode;
}

int gemm_dispatch(const OfbGemmArgs* a, const GemmEpilogue& ep, cudaStream_t stream) {
  if (a->M <= 0 || a->N <= 0 || a->K <= 0) return fail("gemm: empty problem");
  if (a->N % 8 != 0) return fail("gemm: N must be a multiple of 8");
  const int a_mn = a->a_mn_major, b_mn = a->b_mn_major;
  if (few_rows(a) && !a_mn && a->bn == 0 && a->max_ctas == 0 && gemm_mode_2cta() == -1) return gemm_few_rows(a, ep, stream);
  // K-major: dims {K, rows}, row stride ld*2 bytes. MN-major: dims {rows, K}.
  CUtensorMap tmA, tmB;
  int bn = a->bn;
  const int mode2 = gemm_mode_2cta();
  bool two = bn == 512 || (mode2 == 1 && bn == 0);
  // Cost of the three tilings in waves: a wave of the two-SM kernel (74 pairs, 256 x 256) is one unit. Measured over 257 drawn
  // sizes (K from 128 to 8192, all layouts), a wave of 128 x 128 tiles of the one-SM kernel takes 0.7 of it for short K and 0.85
  // for long, one of 128 x 256 tiles 1.2; what decides is that two waves of the small tile cost more than one unit and three more
  // than two (16006 x 304 x 3528: two waves of pairs 53 us, three of 128 x 128 75 us; 3072 x 1024 x 16384: 48 pairs 88 us, 192 tiles
  // of 128 x 128 114 us), while few tiles belong to the small tile (2331 x 768 x 3072: 22 against 29 us).
  const long long tiles2 = (long long)((a->M + 255) / 256) * ((a->N + 255) / 256);
  const long long tiles256 = (long long)((a->M + 127) / 128) * ((a->N + 255) / 256);
  const long long tiles128 = (long long)((a->M + 127) / 128) * ((a->N + 127) / 128);
  const double cost2 = static_cast<double>((tiles2 + 73) / 74);
  const double cost256 = 1.16 * static_cast<double>((tiles256 + 147) / 148), cost128 = 0.72 * static_cast<double>((tiles128 + 147) / 148);
  const double cost1 = cost256 < cost128 ? cost256 : cost128;
  if (mode2 == -1 && bn == 0) {
    // For short K the epilogue takes longer than the main loop, and two one-SM CTAs per SM (short_k below) get through it faster.
    // Where there are tiles for them, up to K = 384 if the epilogue reads or writes more than the result or has GELU in it (with
    // residual 8773 x 6648 x 272 89 against 114 us with pairs, 43046 x 288 x 312 25.5 against 30.3, with GELU 31909 x 656 x 336 38.5
    // against 43.9, 302 x 13864 x 352 20.1 against 24.3; with residual 42572 x 1392 x 408 142 against 129), else up to 256 (with bias 21856 x
    // 1728 x 280 63 against 56 us, with bias and ReLU 25586 x 3896 x 312 124 against 111, 3764 x 6688 x 256 35.8 against 39.7; bare
    // 3704 x 6520 x 200 31.7 against 32.4). Only for a K-major A: with an M-major one (weight gradients) that kernel does not exist; there
    // one-SM tiles win up to K = 256 where the result is bf16 (9472 x 3328 x 136 22.4 against 26.7 us, 8480 x 1296 x 256 15.3
    // against 17.4), pairs where it is fp32 (4248 x 4360 x 168 55.6 against 59).
    // A product with an activation's gradient keeps to pairs from K = 256 on: alone it is the slower one (55296 x 512 x 256 49.5
    // against 47.3 us), but pairs leave registers for the blocks of another stream, and backward passes run beside others (the row
    // update of an embedding beside two such products: 319 against 363 us, the step 3.52 against 3.56 ms).
    const bool rich = ep.aux_out || ep.residual || ep.act == kActGeluErf || ep.act == kActGeluTanh;
    const bool long_enough = a_mn ? ep.out_fp32 || a->K > 256 : a->K > (tiles128 < 2 * 148 || ep.aux_in ? 255 : rich ? 384 : 256);
    // A caller's limit of one CTA leaves no room for a pair.
    two = kDefault2Cta && cost2 <= cost1 && a->N >= 256 && a->M >= 256 && long_enough && a->max_ctas != 1;
  }
  if (mode2 == 0) two = bn == 512;
  // Few K blocks and many tiles: the epilogue is the bottleneck, so run two one-SM CTAs per SM (short ring) instead of one with a
  // deep ring (802816 x 256 x 64: 136 against 228 us); from K = 768 the deep ring wins (2331 x 2304 x 768: 18 against 23 us).
  const bool short_k = !two && a->K <= 512 && bn == 0 && !a_mn && tiles128 >= 2 * 148 && std::getenv("OFB_GEMM_SHORTK_OFF") == nullptr;
  if (two) {
    if (!a_mn) {
      if (get_tensor_map(&tmA, a->A, 2, 2, a->K, a->M, 0, (uint64_t)a->lda * 2, 0, 64, 128, 0, 3)) return -1;
    } else {
      if (get_tensor_map(&tmA, a->A, 2, 2, a->M, a->K, 0, (uint64_t)a->lda * 2, 0, 64, 64, 0, 3)) return -1;
    }
    if (!b_mn) {
      if (get_tensor_map(&tmB, a->B, 2, 2, a->K, a->N, 0, (uint64_t)a->ldb * 2, 0, 64, 128, 0, 3)) return -1;
    } else {
      if (get_tensor_map(&tmB, a->B, 2, 2, a->N, a->K, 0, (uint64_t)a->ldb * 2, 0, 64, 64, 0, 3)) return -1;
    }
    GemmShape shp2{a->M, a->N, a->K, 1};
    int* st2 = device_status_ptr();
    if (!a_mn && !b_mn) return launch_gemm_2cta<0, 0>(tmA, tmB, shp2, ep, st2, a->max_ctas, stream);
    if (!a_mn && b_mn) return launch_gemm_2cta<0, 1>(tmA, tmB, shp2, ep, st2, a->max_ctas, stream);
    if (a_mn && !b_mn) return launch_gemm_2cta<1, 0>(tmA, tmB, shp2, ep, st2, a->max_ctas, stream);
    return launch_gemm_2cta<1, 1>(tmA, tmB, shp2, ep, st2, a->max_ctas, stream);
  }
  if (short_k) bn = 128;
  if (bn != 128 && bn != 256) bn = (cost256 < cost128 && a->N >= 256) ? 256 : 128;
  if (!a_mn) {
    if (get_tensor_map(&tmA, a->A, 2, 2, a->K, a->M, 0, (uint64_t)a->lda * 2, 0, 64, 128, 0, 3)) return -1;
  } else {
    if (get_tensor_map(&tmA, a->A, 2, 2, a->M, a->K, 0, (uint64_t)a->lda * 2, 0, 64, 64, 0, 3)) return -1;
  }
  if (!b_mn) {
    if (get_tensor_map(&tmB, a->B, 2, 2, a->K, a->N, 0, (uint64_t)a->ldb * 2, 0, 64, a_mn ? bn : gemm_b_rows(a->N, bn), 0, 3)) return -1;
  } else {
    if (get_tensor_map(&tmB, a->B, 2, 2, a->N, a->K, 0, (uint64_t)a->ldb * 2, 0, 64, 64, 0, 3)) return -1;
  }
  GemmShape shp{a->M, a->N, a->K, 1};
  // Split-K: few output tiles but a long K (weight gradients: [out, in] = dY^T X over all tokens) would leave most
  // SMs idle. The K range is cut so that about one work unit per SM exists; partial sums are added atomically into
  // the fp32 output, which is cleared first unless the call accumulates anyway.
  {
    static int sm_count = 0, allow = -1;
    if (sm_count == 0) {
      int dev = 0;
      OFB_CUDA_OK(cudaGetDevice(&dev));
      OFB_CUDA_OK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
    }
    if (allow < 0) {
      const char* e = std::getenv("OFB_GEMM_SPLITK");
      allow = e ? std::atoi(e) : 1;
    }
    const bool plain = !ep.bias && !ep.aux_in && !ep.aux_out && !ep.residual && ep.act == 0 && ep.out_fp32;
    const int tiles = ((a->M + 127) / 128) * ((a->N + bn - 1) / bn);
    const int kblocks = (a->K + 63) / 64;
    int cap = a->max_ctas > 0 && a->max_ctas < sm_count ? a->max_ctas : sm_count;
    if (allow && plain && tiles * 2 <= cap && kblocks >= 16) {
      int splits = cap / tiles;
      if (splits > kblocks / 4) splits = kblocks / 4;
      if (splits > 1) {
        shp.splits = splits;
        if (!ep.accumulate)
          OFB_CUDA_OK(cudaMemset2DAsync(ep.C, static_cast<size_t>(ep.ldc) * 4, 0, static_cast<size_t>(a->N) * 4, a->M, stream));
      }
    }
  }
  int* status = device_status_ptr();
  if (short_k && shp.splits <= 1) {
    if (!b_mn) return launch_gemm<128, 0, 0, 2, 2>(tmA, tmB, shp, ep, status, a->max_ctas, stream);
    return launch_gemm<128, 0, 1, 2, 2>(tmA, tmB, shp, ep, status, a->max_ctas, stream);
  }
#define OFB_GEMM_CASE(BN_, AM_, BM_) \
  if (bn == BN_ && a_mn == AM_ && b_mn == BM_) return launch_gemm<BN_, AM_, BM_>(tmA, tmB, shp, ep, status, a->max_ctas, stream);
  OFB_GEMM_CASE(256, 0, 0)
  OFB_GEMM_CASE(256, 0, 1)
  OFB_GEMM_CASE(256, 1, 0)
  OFB_GEMM_CASE(256, 1, 1)
  OFB_GEMM_CASE(128, 0, 0)
  OFB_GEMM_CASE(128, 0, 1)
  OFB_GEMM_CASE(128, 1, 0)
  OFB_GEMM_CASE(128, 1, 1)
#undef OFB_GEMM_CASE
  return fail("gemm: unsupported configuration");
}

}  // namespace ofb

OFB_API int ofb_gemm_bf16(const OfbGemmArgs* a, void* stream) {
  using namespace ofb;
  GemmEpilogue ep;
  std::memset(&ep, 0, sizeof(ep));
  ep.C = a->C;
  ep.ldc = a->ldc;
  ep.bias = reinterpret_cast<const __nv_bfloat16*>(a->bias);
  ep.residual = reinterpret_cast<const __nv_bfloat16*>(a->residual);
  ep.ldr = a->ldr;
  ep.aux_in = reinterpret_cast<const __nv_bfloat16*>(a->aux_in);
  ep.aux_out = reinterpret_cast<__nv_bfloat16*>(a->aux_out);
  ep.ld_aux = a->ld_aux;
  ep.alpha = a->alpha;
  ep.act = a->act;
  ep.out_fp32 = a->out_fp32;
  ep.accumulate = a->accumulate;
  ep.residual_mask = a->residual ? reinterpret_cast<const unsigned char*>(a->residual_mask) : nullptr;
  if (reinterpret_cast<uintptr_t>(ep.residual_mask) & 3) return fail("gemm: the residual's mask must be 4-byte aligned");
  return gemm_dispatch(a, ep, reinterpret_cast<cudaStream_t>(stream));
}

OFB_API const char* ofb_last_error() { return ofb::last_error().c_str(); }

// Reads (and optionally clears) the device status block written by kernels whose bounded
// waits gave up. Synchronises the device: call it at step boundaries, not per kernel.
OFB_API int ofb_read_status(int clear, int* out_code, int* out_detail) {
  int* p = ofb::device_status_ptr();
  if (!p) return ofb::fail("no status block");
  int h[2] = {0, 0};
  OFB_CUDA_OK(cudaMemcpy(h, p, sizeof(h), cudaMemcpyDeviceToHost));
  if (out_code) *out_code = h[0];
  if (out_detail) *out_detail = h[1];
  if (clear && (h[0] || h[1])) OFB_CUDA_OK(cudaMemset(p, 0, 64 * sizeof(int)));
  return 0;
}
