// bf16 GEMM for few rows (M <= 64: tokens of a decoding step, small batches): D[M,N] = epilogue(A[M,K] B[N,K]^T).
//
// What bounds it is reading B once. The tiled kernels give 128 output columns to a CTA, so that N = 4096 occupies 32 of 148 SMs and
// the weights arrive at a fifth of the memory's rate. Here the product is turned round, D^T = B A^T, with 128 rows of B as the
// tensor core's M and the few rows of A as its N (16, 32 or 64: no work on rows that are not there), and the CTAs of a cluster of up to
// eight share the K range of a tile. Their partial sums meet in shared memory: after one cluster barrier every CTA adds its share of
// the tile over the peers' copies and runs the epilogue on it, 8 columns a thread, in 16-byte accesses. No workspace, no atomics,
// the sums in one order.
//
// Per CTA (192 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 move the accumulator to shared memory; all of them
// reduce. About 100 KB of ring: two CTAs per SM, up to 200 KB in flight.
//
// Measured (us a call back to back, weights from memory; tiled kernels / this one / the weights at 6547 GB/s), bias and residual:
//   8 x 12288 x 4096  39.5 / 22.1 / 15.4      8 x 16384 x 4096  42.1 / 27.0 / 20.5      8 x 4096 x 16384  65.7 / 27.7 / 20.5
//   1 x 3072 x 1024   11.7 /  6.2 /  1.0      1 x 1024 x 4096   21.5 /  8.3 /  1.3     64 x 12288 x 4096  30.3 / 26.2 / 15.4
// What is left is the start (two barriers, a cluster, the first loads: 4 us) and, from 33 rows on, the rows' own tiles from L2.
#pragma once
#include "gemm_2cta.cuh"

namespace ofb {

template <int NP>
struct FewRowsCfg {
  static constexpr int BM = 128;                // rows of B per tile
  static constexpr int BK = 64;
  static constexpr int W_BYTES = BM * BK * 2;
  static constexpr int X_BYTES = NP * BK * 2;
  static constexpr int STAGES = NP == 64 ? 4 : 5;
  static constexpr int TMEM_COLS = NP == 64 ? 64 : 32;
  static constexpr int RING_BYTES = STAGES * (W_BYTES + X_BYTES);   // the partial sums take its place: NP x 128 fp32
  static constexpr int SMEM_BYTES = RING_BYTES + 256 + 1024;
  static constexpr int THREADS = 192;
  static_assert(NP * BM * 4 <= RING_BYTES && 2 * (SMEM_BYTES + 1024) <= 228 * 1024, "shared memory");
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void few_rows_unpack(const uint4& q, float (&v)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 few_rows_pack(const float (&v)[8]) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

// The order of operations of gemm_epilogue_chunk, for 8 columns of one row.
__device__ __forceinline__ void few_rows_epilogue(const GemmEpilogue& ep, float (&v)[8], long long row, int col, int n_cols) {
  float h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] *= ep.alpha;
  if (ep.bias) {
    few_rows_unpack(__ldg(reinterpret_cast<const uint4*>(ep.bias + col)), h);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += h[j];
  }
  if (ep.aux_out) *reinterpret_cast<uint4*>(ep.aux_out + row * ep.ld_aux + col) = few_rows_pack(v);
  if (ep.aux_in) {
    few_rows_unpack(*reinterpret_cast<const uint4*>(ep.aux_in + row * ep.ld_aux + col), h);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = ep.act == kActRelu ? (h[j] > 0.f ? v[j] : 0.f) : v[j] * apply_act_grad(h[j], ep.act);
  } else if (ep.act) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = apply_act(v[j], ep.act);
  }
  if (ep.residual) {
    few_rows_unpack(*reinterpret_cast<const uint4*>(ep.residual + row * ep.ldr + col), h);
    const unsigned int keep = ep.residual_mask ? ep.residual_mask[row * (n_cols >> 3) + (col >> 3)] : 0xffu;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += (keep >> j) & 1u ? h[j] : 0.f;
  }
  if (ep.out_fp32) {
    float4* p = reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.C) + row * ep.ldc + col);
    float4 lo = make_float4(v[0], v[1], v[2], v[3]), hi = make_float4(v[4], v[5], v[6], v[7]);
    if (ep.accumulate) {
      const float4 a = p[0], b = p[1];
      lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
      hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
    }
    p[0] = lo;
    p[1] = hi;
  } else {
    uint4* p = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(ep.C) + row * ep.ldc + col);
    uint4 q = few_rows_pack(v);
    if (ep.accumulate) {       // the rounded result is added, as in epi_store_bf16
      few_rows_unpack(q, v);
      few_rows_unpack(*p, h);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += h[j];
      q = few_rows_pack(v);
    }
    *p = q;
  }
}

// Grid: (tiles of 128 columns) x (CTAs per tile), clusters of the latter. W_MN: B is stored [K, N].
template <int NP, int W_MN>
__global__ void __launch_bounds__(192, 2)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, GemmShape shp, GemmEpilogue ep,
                     int* status) {
  using Cfg = FewRowsCfg<NP>;
  constexpr int BM = Cfg::BM, BK = Cfg::BK, STAGES = Cfg::STAGES, W_BYTES = Cfg::W_BYTES, X_BYTES = Cfg::X_BYTES;
  constexpr uint32_t IDESC = make_idesc_bf16(BM, NP, W_MN, 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = smem + STAGES * W_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int parts = shp.splits;
  const int part = static_cast<int>(cluster_ctarank());
  const int n0 = (blockIdx.x / parts) * BM;
  const int kblocks = (shp.K + BK - 1) / BK;
  const int kb_per = (kblocks + parts - 1) / parts;
  const int kb0 = part * kb_per, kb1 = min(kblocks, kb0 + kb_per);   // never empty: the host counts the parts that way

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(&full[stage], W_BYTES + X_BYTES);
        uint8_t* w_dst = sW + stage * W_BYTES;
        if (W_MN) {
#pragma unroll
          for (int c = 0; c < BM / 64; ++c) tma_load_2d(w_dst + c * (BK * 128), &tmW, &full[stage], n0 + c * 64, kb * BK);
        } else {
          tma_load_2d(w_dst, &tmW, &full[stage], kb * BK, n0);
        }
        tma_load_2d(sX + stage * X_BYTES, &tmX, &full[stage], kb * BK, 0);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t w_base = smem_u32(sW + stage * W_BYTES), x_base = smem_u32(sX + stage * X_BYTES);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t dw = W_MN ? make_smem_desc_sw128(w_base + k * 2048, BK * 128, 1024) : make_smem_desc_sw128(w_base + k * 32, 16, 1024);
          const uint64_t dx = make_smem_desc_sw128(x_base + k * 32, 16, 1024);
          umma_bf16_ss(tmem_base, dw, dx, IDESC, (kb != kb0 || k != 0) ? 1u : 0u);
        }
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tfull);
    }
    __syncwarp();
  } else {
    // accumulator (lane = column of the result, TMEM column = row) to shared memory as [row][128]; the products have read the ring
    const int quad = warp & 3;
    float* sums = reinterpret_cast<float*>(smem);
    if (mbar_wait(tfull, 0, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < Cfg::TMEM_COLS / 32; ++c) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + c * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c * 32 + j < NP && c * 32 + j < shp.M) sums[(c * 32 + j) * BM + quad * 32 + lane] = __uint_as_float(r[j]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // every part's sums are in its shared memory

  {
    const uint32_t local = smem_u32(smem);
    const int vecs = shp.M * (BM / 8);               // 8 columns of a row each
    for (int i = part * Cfg::THREADS + threadIdx.x; i < vecs; i += parts * Cfg::THREADS) {
      const int m = i / (BM / 8), c = (i % (BM / 8)) * 8;
      if (n0 + c >= shp.N) continue;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
      // all peers' sums are asked for before the first is added
      float4 lo[8], hi[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        if (p < parts) {
          const uint32_t a = map_to_cta(local + (m * BM + c) * 4, p);
          lo[p] = ld_cluster_f4(a);
          hi[p] = ld_cluster_f4(a + 16);
        }
      }
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        if (p < parts) {
          v[0] += lo[p].x; v[1] += lo[p].y; v[2] += lo[p].z; v[3] += lo[p].w;
          v[4] += hi[p].x; v[5] += hi[p].y; v[6] += hi[p].z; v[7] += hi[p].w;
        }
      }
      few_rows_epilogue(ep, v, m, n0 + c, shp.N);
    }
  }
  cluster_sync_all();      // nobody leaves while a peer may read its sums
  tc_fence_after();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, (int)kStatusMbarTimeout);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

}  // namespace ofb
