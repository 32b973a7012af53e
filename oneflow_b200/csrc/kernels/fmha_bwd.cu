// Fused multi-head attention backward for sm_100a (bf16, head dim 64 or 128; query length != key length,
// grouped-query attention and Philox dropout as in the forward kernel).
//
// A CTA works on one 128-key tile at a time (K_j, V_j stay resident in shared memory) of one (batch, key/value head)
// and walks over the query tiles i that see it, for every query head of the group in turn (so dK and dV of a
// shared key/value head accumulate in TMEM and need no second reduction). Per (i, j) pair five tcgen05 products run,
// all fed from the same shared-memory tiles without any transposition pass. The scores are formed transposed (TMEM lane =
// key row), so that P^T is the A operand of dV straight from the TMEM columns it was computed in:
//     S^T  = K_j Q_i^T           (K-major  x K-major)       -> TMEM, P^T (bf16) is written over it
//     dP^T = V_j dO_i^T          (K-major  x K-major)       -> TMEM
//     dV  += P^T dO_i            (TMEM     x MN-major)      -> TMEM accumulator
//     dK  += dS^T Q_i            (K-major  x MN-major)      -> TMEM accumulator
//     dQ_i partial = dS K_j      (MN-major x MN-major)      -> TMEM, staged in shared memory and added to HBM by TMA
// Roles (512 threads): warp 0 TMA producer, warp 1 tcgen05 issuer, warps 2 / 3 fetch log-sum-exp / delta of the next query
// tile, warps 4..7 drain dQ, warps 8..15 form P and dS: one thread owns one key row, warps 8..11 its first 64 query
// columns, warps 12..15 the other 64.
// The products of neighbouring pairs are interleaved: S of pair i + 1 is issued behind dV of pair i (products of one thread
// run in order, so the columns of P are free by then), hence the exponentials of pair i + 1 run while dQ, dK of pair i and
// dP of pair i + 1 are multiplied and dQ is drained. The chain that remains between two pairs is dS -> dQ -> drain -> dP
// (at D = 128 dQ has no TMEM columns of its own and takes those of dP).
// At D = 64 there is room for the K and V of two key tiles: the scores of the next one are there when this one's gradients have
// left TMEM.
// What bounds it: at D = 128 shared-memory bandwidth (per pair the products read 288 KiB of operands, staging dS and dQ and
// the copies of Q, dO and dQ move 224 KiB: 4100 clocks, the products themselves 2560), the fp32 reductions of dQ in L2, and on long
// sequences the power limit; at D = 64 the threads that form P and dS (1310 and 1000 clocks of 2700 a pair, products 1280) and, with
// four pairs a key tile, the 4000 clocks between two key tiles.
// The grid has one CTA per key tile, but a running CTA takes over the next one that has not started (cluster launch control), so
// that barriers, TMEM and the first loads of a tile do not wait for the end of the one before; the order stays the hardware's.
// Measured on a B200, this kernel alone (in brackets with a mask test in every group of four exponentials, dS stored behind the
// last of them, and dK and dV written a row per thread): batch 4, 32 heads, 2048 x 2048, D = 128, causal 340 us (368); batch 1, 32 / 8
// heads, 8192 x 8192, D = 128, causal 1377 us (1379); batch 32, 16 heads, 512 x 512, D = 64 126 us (152); batch 8, 16 heads,
// 500 x 1100, D = 64 70.5 us (86.9); batch 3, 12 heads, 777 x 777, D = 64, causal 20.2 us (24.5).
// TMEM: S/P | dP (D = 128: also dQ) | dV | dK | D = 64: dQ.
//
// Reference counterpart: oneflow/user/kernels/scaled_dot_product_attention_grad_kernel.cu
// (flash-attention library call).
#include <type_traits>

#include "../common/host_utils.h"
#include "../common/philox.cuh"
#include "../common/ptx.cuh"
#include "ofb_kernels.h"

namespace ofb {

int fmha_tensor_map(CUtensorMap* out, const void* ptr, int B, int S, int H, int D, long long row_stride);
int fmha_dropout_cfg(DropoutCfg* d, float p_dropout, unsigned long long seed, unsigned int offset);

struct FmhaBwdParams {
  const float* lse;     // [B, H, Sq]
  const float* delta;   // [B, H, Sq] rowsum(dO * O)
  float* dq_acc;        // [B, Sq, H, D] fp32, zero-initialised, receives red.add
  __nv_bfloat16* dk;    // element (b,s,hk,d) at ((b*Sk+s)*dkv_row_stride + hk*D + d)
  __nv_bfloat16* dv;
  long long dkv_row_stride;
  const int* kv_len;
  int B, H, Hk, Sq, Sk, D;
  int causal;
  int causal_off;       // Sk - Sq
  DropoutCfg drop;
  float scale;          // softmax scale
  float scale_log2e;
  int n_kt;             // key tiles of one head
  int chunk;            // heads (of B * Hk) that are walked together, key tiles with the most query tiles first
  int* status;
};

template <int D>
struct FmhaBwdCfg {
  static constexpr int T_BYTES = 128 * D * 2;            // one [128 x D] tile
  static constexpr int DO_STAGES = D == 128 ? 1 : 2;     // at D = 128 shared memory has room for one dO tile
  static constexpr int KV_STAGES = D == 128 ? 1 : 2;     // and for the K and V of one key tile
  static constexpr int DS_BYTES = 128 * 128 * 2;
  static constexpr int SLAB_BYTES = 128 * 32 * 4;        // 32 columns of dQ in fp32, two of them in flight
  static constexpr int STAT_BYTES = 2 * 2 * 128 * 4;     // log-sum-exp and delta of two query tiles
  // no slack for aligning by hand: the dynamic shared memory starts the CTA's window (checked by the kernel)
  static constexpr int BAR_BYTES = 288;                  // 30 mbarriers, TMEM slot, abort flag, two answers of 16 bytes
  static constexpr int SMEM_BYTES = (2 * KV_STAGES + 2 + DO_STAGES) * T_BYTES + DS_BYTES + 2 * SLAB_BYTES + STAT_BYTES + BAR_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};

// fp32 add-reduction of a shared-memory tile into global memory through TMA (one bulk operation instead of
// thousands of per-thread red instructions; L2 sees whole 128-byte lines).
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, const void* smem_src, int x, int y, int z, int w) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
template <int D, bool DROP>
__global__ void __launch_bounds__(512, 1)
fmha_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, FmhaBwdParams p) {
  using Cfg = FmhaBwdCfg<D>;
  constexpr int DCH = D / 64, DO_ST = Cfg::DO_STAGES, KV_ST = Cfg::KV_STAGES;
  constexpr int CH_BYTES = 128 * 128;
  constexpr bool kOwnDq = D == 64;                                // dQ has TMEM columns of its own
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);   // S^T, dP^T
  constexpr uint32_t IDESC_KV = make_idesc_bf16(128, D, 0, 1);    // dV (A in TMEM), dK (A K-major); B MN-major
  constexpr uint32_t IDESC_DQ = make_idesc_bf16(128, D, 1, 1);    // dQ: both operands MN-major

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {   // uniform over the CTA: nobody has touched a barrier or TMEM yet
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, (int)kStatusBounds);
    return;
  }
  uint8_t* sK = smem;                               // KV_ST stages
  uint8_t* sV = sK + KV_ST * Cfg::T_BYTES;          // KV_ST stages
  uint8_t* sQ = sV + KV_ST * Cfg::T_BYTES;          // 2 stages
  uint8_t* sdO = sQ + 2 * Cfg::T_BYTES;             // DO_ST stages
  uint8_t* sdS = sdO + DO_ST * Cfg::T_BYTES;        // dS^T: two 64-query chunks of [128 keys x 128 bytes]
  uint8_t* sStage = sdS + Cfg::DS_BYTES;            // two dQ slabs
  float* sStat = reinterpret_cast<float*>(sStage + 2 * Cfg::SLAB_BYTES);   // [stage][-lse | -delta][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStat) + Cfg::STAT_BYTES);
  uint64_t* k_full = bars;          // [2]
  uint64_t* v_full = bars + 2;      // [2]
  uint64_t* kv_empty = bars + 4;    // [2] every product of a key tile has finished
  uint64_t* q_full = bars + 6;      // [2]
  uint64_t* q_empty = bars + 8;     // [2]
  uint64_t* do_full = bars + 10;    // [2]
  uint64_t* do_empty = bars + 12;   // [2]
  uint64_t* stat_full = bars + 14;  // [2] 64 fetching threads
  uint64_t* stat_empty = bars + 16; // [2] 8 compute warps
  uint64_t* next_full = bars + 18;  // [2] the answer that names the CTA's next key tile
  uint64_t* next_empty = bars + 20; // [2] 16 warps
  uint64_t* s_full = bars + 22;
  uint64_t* p_ready = bars + 23;    // 256
  uint64_t* dp_full = bars + 24;
  uint64_t* ds_ready = bars + 25;   // 256
  uint64_t* dq_full = bars + 26;
  uint64_t* dq_drained = bars + 27; // 128
  uint64_t* all_done = bars + 28;
  uint64_t* acc_free = bars + 29;   // 256: dK and dV have left TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 30);
  uint8_t* answers = reinterpret_cast<uint8_t*>(bars + 32);   // [2] 16 bytes
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Key tile number `item`: heads in chunks whose queries, gradients and dQ accumulators stay in L2 together; inside a chunk the
  // key tiles that most query tiles see (the first ones) come first, so that the short ones fill the tail.
  const int group = p.H / p.Hk;          // query heads per key/value head
  const int n_qt = (p.Sq + 127) / 128;
  struct Item {
    int hk, b, k0, kv_limit;
    int i_start;   // first query tile with a row that sees this key tile: row + causal_off >= k0
    int n_iter;    // pairs: query tiles i_start .. n_qt - 1 of every head of the group
  };
  auto item_of = [&](int item) {
    const int in_chunk_max = p.chunk * p.n_kt;
    const int ck = item / in_chunk_max, rem = item % in_chunk_max;
    const int heads_here = min(p.chunk, p.B * p.Hk - ck * p.chunk);
    const int bhk = ck * p.chunk + rem % heads_here;
    Item it;
    it.hk = bhk % p.Hk;
    it.b = bhk / p.Hk;
    it.k0 = rem / heads_here * 128;
    it.kv_limit = p.kv_len ? min(p.Sk, p.kv_len[it.b]) : p.Sk;
    it.i_start = p.causal ? max(0, it.k0 - p.causal_off) / 128 : 0;
    it.n_iter = it.k0 < it.kv_limit ? max(0, n_qt - it.i_start) * group : 0;
    return it;
  };
  // The CTA works through key tiles until none is left: every role walks the same sequence. `n` counts the tiles.
  auto next_item = [&](int n, int& item) -> bool {      // called by whole warps
    const bool ok = mbar_wait(&next_full[n & 1], (n >> 1) & 1, abort_flag);
    int nx = 0;
    const bool more = ok && clc_take(answers + (n & 1) * 16, nx);
    item = nx;
    __syncwarp();
    if (lane == 0) mbar_arrive(&next_empty[n & 1]);
    return more;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&kv_empty[s], 1);
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
      mbar_init(&stat_full[s], 64);
      mbar_init(&stat_empty[s], 8);
    }
    mbar_init(s_full, 1);
    mbar_init(p_ready, 256);
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, 256);
    mbar_init(dq_full, 1);
    mbar_init(dq_drained, 128);
    mbar_init(all_done, 1);
    mbar_init(acc_free, 256);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&next_full[s], 1);
      mbar_init(&next_empty[s], 16);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
    tma_prefetch_desc(&tmdQ);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base;          // P^T of query columns 0..63 over columns 0..31, of 64..127 over columns 64..95
  const uint32_t tdP = tmem_base + 128;
  const uint32_t tdV = tmem_base + 256;
  const uint32_t tdK = tmem_base + 256 + D;
  const uint32_t tdQ = kOwnDq ? tmem_base + 256 + 2 * D : tdP;

  // registers: 512 threads x 128 at launch = 4 warpgroups x 128 on average; the drain warps hold D columns of dQ each
  constexpr int kRegsControl = D == 64 ? 80 : 64, kRegsDrain = D == 64 ? 112 : 144, kRegsCompute = D == 64 ? 160 : 152;
  static_assert(kRegsControl + kRegsDrain + 2 * kRegsCompute == 512, "a split above the launch's registers would wait for ever");
  if (warp < 4) {
    reg_dec<kRegsControl>();
    int item = blockIdx.x;
    int g0 = 0;        // pairs of the tiles before this one: pair t of this tile is number g0 + t, which gives slots and phases
    int act = 0;       // tiles before this one that had any pair
    bool ok = true;
    for (int n = 0;; ++n) {
      const Item it = item_of(item);
      if (warp == 0) {
        if (elect_one()) {
          // Ask for the next tile a few pairs before the loads of this one end: early enough for the answer to be there, late
          // enough that long tiles do not bind another one at their start (that cost 14 % at 512 causal tiles of 46 to 256 pairs).
          auto ask = [&]() {      // both slots' readers of two tiles ago are done
            if (!mbar_wait(&next_empty[n & 1], ((n >> 1) & 1) ^ 1, abort_flag)) return;
            fence_proxy_async_smem();
            clc_ask(answers + (n & 1) * 16, &next_full[n & 1]);
          };
          const int ask_at = max(0, it.n_iter - 4);
          if (it.n_iter == 0 || !ok) ask();
          if (it.n_iter > 0 && ok) {
            auto load = [&](uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int head, int row) {
              mbar_arrive_expect_tx(bar, Cfg::T_BYTES);
#pragma unroll
              for (int c = 0; c < DCH; ++c) tma_load_4d(dst + c * CH_BYTES, m, bar, c * 64, head, row, it.b);
            };
            int h = it.hk * group, i = it.i_start;
            for (int t = 0; t < it.n_iter; ++t) {
              const int g = g0 + t, st = g & 1, sd = g % DO_ST;
              if (t == ask_at) ask();
              if (!mbar_wait(&q_empty[st], ((g >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
              load(sQ + st * Cfg::T_BYTES, &tmQ, &q_full[st], h, i * 128);
              if (t == 0) {
                const int kv = act % KV_ST;
                if (!mbar_wait(&kv_empty[kv], ((act / KV_ST) & 1) ^ 1, abort_flag)) { ok = false; break; }
                load(sK + kv * Cfg::T_BYTES, &tmK, &k_full[kv], it.hk, it.k0);
                load(sV + kv * Cfg::T_BYTES, &tmV, &v_full[kv], it.hk, it.k0);
              }
              if (!mbar_wait(&do_empty[sd], ((g / DO_ST) & 1) ^ 1, abort_flag)) { ok = false; break; }
              load(sdO + sd * Cfg::T_BYTES, &tmdO, &do_full[sd], h, i * 128);
              if (++i == n_qt) { i = it.i_start; ++h; }
            }
          }
        }
        __syncwarp();
      } else if (warp == 1) {
        if (elect_one() && it.n_iter > 0 && ok) {
          const int kv = act % KV_ST;
          const uint32_t kv_ph = (act / KV_ST) & 1;
          const uint32_t k_base = smem_u32(sK + kv * Cfg::T_BYTES), v_base = smem_u32(sV + kv * Cfg::T_BYTES), ds_base = smem_u32(sdS);
          auto kk_off = [](int kk) -> uint32_t { return (kk >> 2) * CH_BYTES + (kk & 3) * 32; };   // K-major step of 16
          auto issue_s = [&](int g) {
            const uint32_t q_base = smem_u32(sQ + (g & 1) * Cfg::T_BYTES);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              umma_bf16_ss(tS, make_smem_desc_sw128(k_base + kk_off(kk), 16, 1024), make_smem_desc_sw128(q_base + kk_off(kk), 16, 1024),
                           IDESC_S, kk != 0 ? 1u : 0u);
            umma_commit(s_full);
          };
          // dP^T of pair g: its columns are free once dS of the pair before was read (that pair's dQ waited for it) and, at
          // D = 128, the dQ in them was drained
          auto issue_dp = [&](int g) -> bool {
            if (!mbar_wait(&do_full[g % DO_ST], (g / DO_ST) & 1, abort_flag)) return false;
            if (!kOwnDq && g > 0 && !mbar_wait(dq_drained, (g - 1) & 1, abort_flag)) return false;
            tc_fence_after();
            const uint32_t do_base = smem_u32(sdO + (g % DO_ST) * Cfg::T_BYTES);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              umma_bf16_ss(tdP, make_smem_desc_sw128(v_base + kk_off(kk), 16, 1024), make_smem_desc_sw128(do_base + kk_off(kk), 16, 1024),
                           IDESC_S, kk != 0 ? 1u : 0u);
            umma_commit(dp_full);
            return true;
          };
          ok = mbar_wait(&k_full[kv], kv_ph, abort_flag) && mbar_wait(&q_full[g0 & 1], (g0 >> 1) & 1, abort_flag);
          if (ok) { tc_fence_after(); issue_s(g0); }
          ok = ok && mbar_wait(&v_full[kv], kv_ph, abort_flag);
          ok = ok && issue_dp(g0);
          // the accumulators of the tile before have left TMEM
          ok = ok && mbar_wait(acc_free, (act & 1) ^ 1, abort_flag);
          for (int t = 0; t < it.n_iter && ok; ++t) {
            const int g = g0 + t;
            const uint32_t ph = g & 1;
            const uint32_t q_base = smem_u32(sQ + (g & 1) * Cfg::T_BYTES);
            const uint32_t do_base = smem_u32(sdO + (g % DO_ST) * Cfg::T_BYTES);
            // dV += P^T dO_i
            if (!mbar_wait(p_ready, ph, abort_flag)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_bf16_ts(tdV, tS + (kk >> 2) * 64 + (kk & 3) * 8, make_smem_desc_sw128(do_base + kk * 2048, CH_BYTES, 1024), IDESC_KV,
                           (t | kk) != 0 ? 1u : 0u);
            umma_commit(&do_empty[g % DO_ST]);   // dP of this pair was issued before
            // S^T of the next pair, over the P that dV has read by then
            if (t + 1 < it.n_iter) {
              if (!mbar_wait(&q_full[(g + 1) & 1], ((g + 1) >> 1) & 1, abort_flag)) { ok = false; break; }
              tc_fence_after();
              issue_s(g + 1);
            }
            // dQ partial = dS K_j, then dK += dS^T Q_i while dQ is drained
            if (!mbar_wait(ds_ready, ph, abort_flag)) { ok = false; break; }
            if (kOwnDq && g > 0 && !mbar_wait(dq_drained, (g - 1) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_bf16_ss(tdQ, make_smem_desc_sw128(ds_base + kk * 2048, CH_BYTES, 1024),
                           make_smem_desc_sw128(k_base + kk * 2048, CH_BYTES, 1024), IDESC_DQ, kk != 0 ? 1u : 0u);
            umma_commit(dq_full);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_bf16_ss(tdK, make_smem_desc_sw128(ds_base + kk_off(kk), 16, 1024),
                           make_smem_desc_sw128(q_base + kk * 2048, CH_BYTES, 1024), IDESC_KV, (t | kk) != 0 ? 1u : 0u);
            umma_commit(&q_empty[g & 1]);
            if (t + 1 < it.n_iter && !issue_dp(g + 1)) { ok = false; break; }
          }
          if (ok) {
            umma_commit(all_done);
            umma_commit(&kv_empty[kv]);
          }
        }
        __syncwarp();
      } else if (it.n_iter > 0 && ok) {
        // warp 2: minus log-sum-exp in log2 units, -inf where the row does not exist or saw no key (P becomes 0); warp 3: -delta
        int h = it.hk * group, i = it.i_start;
        for (int t = 0; t < it.n_iter; ++t) {
          const int g = g0 + t, st = g & 1;
          float val[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = i * 128 + lane * 4 + e;
            const long long idx = (static_cast<long long>(it.b) * p.H + h) * p.Sq + row;
            if (warp == 2) {
              const float l = row < p.Sq ? p.lse[idx] : -INFINITY;
              val[e] = l == -INFINITY ? -INFINITY : l * -1.4426950408889634f;
            } else {
              val[e] = row < p.Sq ? -p.delta[idx] : 0.f;
            }
          }
          if (!mbar_wait(&stat_empty[st], ((g >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          *reinterpret_cast<float4*>(sStat + (st * 2 + (warp - 2)) * 128 + lane * 4) = make_float4(val[0], val[1], val[2], val[3]);
          mbar_arrive(&stat_full[st]);
          if (++i == n_qt) { i = it.i_start; ++h; }
        }
        __syncwarp();
      }
      g0 += it.n_iter;
      act += it.n_iter > 0;
      if (!next_item(n, item)) break;
    }
  } else if (warp < 8) {
    if constexpr (D == 64) reg_dec<kRegsDrain>();
    else reg_inc<kRegsDrain>();
    // Drain the dQ partials: TMEM -> swizzled fp32 staging slabs -> one TMA add-reduction per 32 columns into the accumulator.
    // Every warp stages and reduces its own 32 rows, so no warp waits for another. (All 128 threads meeting around one
    // 128-row reduction per slab: 1.78 instead of 1.47 ms for batch 1, 32 / 8 heads, 8192 x 8192, D = 128, causal.)
    const int quad = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    int item = blockIdx.x, g0 = 0;
    bool ok = true;
    for (int n = 0;; ++n) {
      const Item it = item_of(item);
      int h = it.hk * group, i = it.i_start;
      for (int t = 0; t < it.n_iter && ok; ++t) {
        if (!mbar_wait(dq_full, (g0 + t) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        // the whole partial leaves TMEM before anything else happens: the next dP waits for these columns at D = 128
        uint32_t v[D / 32][32];
        __syncwarp();
#pragma unroll
        for (int s = 0; s < D / 32; ++s) tmem_ld_32x32(tdQ + lane_addr + s * 32, v[s]);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(dq_drained);
        if (i * 128 + quad * 32 < p.Sq) {   // a box may hang over the last row, but does not start behind it
#pragma unroll
          for (int s = 0; s < D / 32; ++s) {
            if (lane == 0) tma_store_wait_read<1>();     // the reduction before the last has read this slab
            __syncwarp();
            uint8_t* st = sStage + (s & 1) * Cfg::SLAB_BYTES + quad * 4096;
#pragma unroll
            for (int g = 0; g < 8; ++g)
              *reinterpret_cast<uint4*>(st + lane * 128 + ((g ^ (lane & 7)) << 4)) =
                  make_uint4(v[s][4 * g], v[s][4 * g + 1], v[s][4 * g + 2], v[s][4 * g + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_reduce_add_4d(&tmdQ, st, s * 32, h, i * 128 + quad * 32, it.b);
              tma_store_commit();
            }
          }
        }
        if (++i == n_qt) { i = it.i_start; ++h; }
      }
      __syncwarp();
      g0 += it.n_iter;
      if (!next_item(n, item)) break;
    }
    if (lane == 0) tma_store_wait<0>();
    __syncwarp();
  } else {
    reg_inc<kRegsCompute>();
    const int quad = warp & 3;
    const int half = (warp - 8) >> 2;          // which 64 query columns of every tile this thread takes
    const int r = quad * 32 + lane;            // key row of the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    int item = blockIdx.x, g0 = 0, act = 0;
    bool ok = true;
    for (int n = 0;; ++n) {
      const Item it = item_of(item);
      const int krow = it.k0 + r;
      if (it.n_iter > 0) {
        uint8_t* ds_row = sdS + half * CH_BYTES + r * 128;   // this half's 64 queries = one swizzled chunk
        const uint32_t tSh = tS + lane_addr + half * 64, tdPh = tdP + lane_addr + half * 64;
        const uint64_t scale2 = pack_f32x2(__float_as_uint(p.scale_log2e), __float_as_uint(p.scale_log2e));
        int h = it.hk * group, i = it.i_start;
        for (int t = 0; t < it.n_iter && ok; ++t) {
          const int g = g0 + t;
          const uint32_t ph = g & 1;
          const int st = g & 1;
          const int q0 = i * 128;
          const float* nlse = sStat + st * 256 + half * 64;
          const float* ndelta = nlse + 128;
          const bool need_mask = (p.causal && it.k0 + 127 > q0 + p.causal_off) || (it.k0 + 128 > it.kv_limit);
          // first visible query column of this thread's half
          const int c_min = krow >= it.kv_limit ? 64 : (p.causal ? krow - p.causal_off - q0 - half * 64 : 0);
          uint32_t pk[32];  // P as packed bf16 pairs of this key row's 64 queries
          uint32_t keep_bits[DROP ? 2 : 1];  // dropout: bit c of word w = query column 32 * w + c of this half is kept
          if constexpr (DROP) {
            // a Philox draw covers four neighbouring keys of one query: the four lanes that own them draw a quarter each
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              uint32_t bits = 0;
#pragma unroll
              for (int g4 = 0; g4 < 8; ++g4) {
                const uint32_t row = static_cast<uint32_t>(q0 + half * 64 + w * 32 + g4 * 4 + (lane & 3));
                const uint32_t k4 = dropout_keep4(p.drop, static_cast<uint32_t>(it.b * p.H + h), row, static_cast<uint32_t>(krow >> 2));
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  bits |= ((__shfl_sync(0xffffffffu, k4, (lane & ~3) + e) >> (krow & 3)) & 1u) << (g4 * 4 + e);
              }
              keep_bits[w] = bits;
            }
          }
          if (!mbar_wait(&stat_full[st], (g >> 1) & 1, abort_flag)) { ok = false; break; }
          if (!mbar_wait(s_full, ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          {
            uint32_t v[2][32];
            __syncwarp();
            tmem_ld_32x32(tSh, v[0]);
            tmem_ld_32x32(tSh + 32, v[1]);
            tmem_wait_ld();
            // one straight piece of code per kind of tile: with the test inside, every four elements were a block of their own and
            // waited for their own loads and exponentials (1650 clocks a pair instead of 1310; the exponentials alone are 1024)
            auto form_p = [&](auto masked) {
#pragma unroll
              for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int e = 0; e < 32; e += 4) {
                  const float4 l4 = *reinterpret_cast<const float4*>(nlse + c * 32 + e);
                  float x[4];
                  unpack_f32x2(fma_f32x2(pack_f32x2(v[c][e], v[c][e + 1]), scale2, pack_f32x2(__float_as_uint(l4.x), __float_as_uint(l4.y))),
                               x[0], x[1]);
                  unpack_f32x2(fma_f32x2(pack_f32x2(v[c][e + 2], v[c][e + 3]), scale2, pack_f32x2(__float_as_uint(l4.z), __float_as_uint(l4.w))),
                               x[2], x[3]);
#pragma unroll
                  for (int k = 0; k < 4; ++k) x[k] = fast_exp2(x[k]);
                  if constexpr (decltype(masked)::value) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                      if (c * 32 + e + k < c_min) x[k] = 0.f;
                  }
                  pk[c * 16 + (e >> 1)] = pack_bf16x2(x[0], x[1]);
                  pk[c * 16 + (e >> 1) + 1] = pack_bf16x2(x[2], x[3]);
                }
              }
            };
            if (need_mask) form_p(std::true_type());
            else form_p(std::false_type());
            // Publish P^T (with dropout: only the kept probabilities, which is what multiplied V in the forward; the factor
            // 1 / keep is applied to dV at the end). Only this thread reads these TMEM columns of S, and it has.
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t w16[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                w16[e] = pk[c * 16 + e];
                if constexpr (DROP)
                  w16[e] &= ((keep_bits[c] >> (2 * e)) & 1u ? 0x0000FFFFu : 0u) | ((keep_bits[c] >> (2 * e + 1)) & 1u ? 0xFFFF0000u : 0u);
              }
              tmem_st_32x16(tSh + c * 16, w16);
            }
            tmem_wait_st();
          }
          tc_fence_before();
          mbar_arrive(p_ready);
          // dS = P * (dP - delta); the softmax scale is applied to the finished dK and dQ. dP of this pair was issued behind dQ and
          // dK of the one before: those have read the last dS when it arrives, and every 16 bytes are stored as they are formed
          if (!mbar_wait(dp_full, ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          {
            uint32_t v[2][32];
            __syncwarp();
            tmem_ld_32x32(tdPh, v[0]);
            tmem_ld_32x32(tdPh + 32, v[1]);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int e = 0; e < 32; e += 8) {
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const int f = e + 4 * u;
                  const float4 nd = *reinterpret_cast<const float4*>(ndelta + c * 32 + f);
                  if constexpr (DROP) {   // the gradient reaches P only through the kept entries, scaled by 1 / keep
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                      v[c][f + k] = (keep_bits[c] >> (f + k)) & 1u ? __float_as_uint(__uint_as_float(v[c][f + k]) * p.drop.inv_keep) : 0u;
                  }
                  const uint32_t w0 = pk[c * 16 + (f >> 1)], w1 = pk[c * 16 + (f >> 1) + 1];
                  float d[4];
                  unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(v[c][f], v[c][f + 1]), pack_f32x2(__float_as_uint(nd.x), __float_as_uint(nd.y))),
                                         pack_f32x2(w0 << 16, w0 & 0xFFFF0000u)), d[0], d[1]);
                  unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(v[c][f + 2], v[c][f + 3]), pack_f32x2(__float_as_uint(nd.z), __float_as_uint(nd.w))),
                                         pack_f32x2(w1 << 16, w1 & 0xFFFF0000u)), d[2], d[3]);
                  w[2 * u] = pack_bf16x2(d[0], d[1]);
                  w[2 * u + 1] = pack_bf16x2(d[2], d[3]);
                }
                *reinterpret_cast<uint4*>(ds_row + (((c * 4 + (e >> 3)) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
              }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&stat_empty[st]);
          fence_proxy_async_smem();
          tc_fence_before();
          mbar_arrive(ds_ready);
          if (++i == n_qt) { i = it.i_start; ++h; }
        }
        // dK (the first half's warps) and dV (the second's) of this key tile: TMEM lane = key row. A warp turns its 32 rows through
        // its own part of dS, which every product has read by now, so that eight lanes write 128 bytes of a row together. (A thread
        // writing its own row, 16 bytes in a line of its own per lane and store, kept the next tile waiting for 3500 clocks.)
        if (ok) ok = mbar_wait(all_done, act & 1, abort_flag);
        if (ok) {
          tc_fence_after();
          const uint32_t src = (half == 0 ? tdK : tdV) + lane_addr;
          __nv_bfloat16* dst = (half == 0 ? p.dk : p.dv) + (static_cast<long long>(it.b) * p.Sk + it.k0 + quad * 32) * p.dkv_row_stride + it.hk * D;
          const float osc = half == 0 ? p.scale : (DROP ? p.drop.inv_keep : 1.f);
          const int rows_here = p.Sk - it.k0 - quad * 32;
#pragma unroll
          for (int c = 0; c < DCH; ++c) {
            uint32_t v[2][32];
            __syncwarp();
            tmem_ld_32x32(src + c * 64, v[0]);
            tmem_ld_32x32(src + c * 64 + 32, v[1]);
            tmem_wait_ld();
            if (c == DCH - 1) {
              tc_fence_before();
              mbar_arrive(acc_free);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const uint32_t* x = v[e >> 2] + (e & 3) * 8;
              *reinterpret_cast<uint4*>(ds_row + ((e ^ (r & 7)) << 4)) =
                  make_uint4(pack_bf16x2(__uint_as_float(x[0]) * osc, __uint_as_float(x[1]) * osc),
                             pack_bf16x2(__uint_as_float(x[2]) * osc, __uint_as_float(x[3]) * osc),
                             pack_bf16x2(__uint_as_float(x[4]) * osc, __uint_as_float(x[5]) * osc),
                             pack_bf16x2(__uint_as_float(x[6]) * osc, __uint_as_float(x[7]) * osc));
            }
            __syncwarp();
            const uint8_t* warp_rows = sdS + half * CH_BYTES + quad * 32 * 128;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int row = e * 4 + (lane >> 3), ch = lane & 7;
              const uint4 q = *reinterpret_cast<const uint4*>(warp_rows + row * 128 + ((ch ^ (row & 7)) << 4));
              if (row < rows_here) *reinterpret_cast<uint4*>(dst + row * p.dkv_row_stride + c * 64 + ch * 8) = q;
            }
            __syncwarp();
          }
        }
      } else if (krow < p.Sk) {
        // Key tile invisible to every query (beyond kv_len, or right of the causal diagonal for all rows): zero gradients.
        __nv_bfloat16* dk_row = p.dk + (static_cast<long long>(it.b) * p.Sk + krow) * p.dkv_row_stride + it.hk * D;
        __nv_bfloat16* dv_row = p.dv + (static_cast<long long>(it.b) * p.Sk + krow) * p.dkv_row_stride + it.hk * D;
        for (int i = half * (D / 2); i < (half + 1) * (D / 2); i += 8) {
          *reinterpret_cast<uint4*>(dk_row + i) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(dv_row + i) = make_uint4(0, 0, 0, 0);
        }
      }
      g0 += it.n_iter;
      act += it.n_iter > 0;
      __syncwarp();
      if (!next_item(n, item)) break;
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, (int)kStatusMbarTimeout);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// delta[b,h,s] = sum_d dO[b,s,h,d] * O[b,s,h,d], and the same elements of the fp32 dQ accumulator are cleared. D / 8 lanes
// share a row, 16 bytes of each operand per lane (one warp per row with 4-byte loads took 49 us where this and a memset of
// the accumulator move 134 MB: batch 32, 16 heads, 512 rows, D = 64).
template <int D>
__global__ void fmha_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, float* __restrict__ delta,
                                  float* __restrict__ dq_acc, int B, int S, int H) {
  constexpr int L = D / 8;             // lanes per row
  const long long total = static_cast<long long>(B) * S * H;
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x % L;
  const bool live = w < total;
  float acc = 0.f;
  if (live) {
    const long long off = w * D + sub * 8;
    const uint4 a = *reinterpret_cast<const uint4*>(o + off);
    const uint4 c = *reinterpret_cast<const uint4*>(d_o + off);
    const uint32_t pa[4] = {a.x, a.y, a.z, a.w}, pc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_bf16x2(pa[e]), y = unpack_bf16x2(pc[e]);
      acc = fmaf(x.x, y.x, acc);
      acc = fmaf(x.y, y.y, acc);
    }
    *reinterpret_cast<float4*>(dq_acc + off) = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(dq_acc + off + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int m = L / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (live && sub == 0) {
    const int h = static_cast<int>(w % H);
    const long long bs = w / H;
    delta[(bs / S * H + h) * S + bs % S] = acc;
  }
}

// dq (bf16, strided rows) = scale * dq_acc (fp32 [B*S, H*D])
__global__ void fmha_dq_cast_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long long rows, int hd,
                                    long long row_stride, float scale) {
  const int vec_per_row = hd >> 3;
  const long long total = rows * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / vec_per_row;
    const int c = static_cast<int>(i % vec_per_row) * 8;
    const float4 a = *reinterpret_cast<const float4*>(acc + row * hd + c);
    const float4 bb = *reinterpret_cast<const float4*>(acc + row * hd + c + 4);
    *reinterpret_cast<uint4*>(dq + row * row_stride + c) =
        make_uint4(pack_bf16x2(a.x * scale, a.y * scale), pack_bf16x2(a.z * scale, a.w * scale), pack_bf16x2(bb.x * scale, bb.y * scale),
                   pack_bf16x2(bb.z * scale, bb.w * scale));
  }
}

template <int D, bool DROP>
static int launch_fmha_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                           const CUtensorMap& tdq, FmhaBwdParams p, cudaStream_t stream) {
  using Cfg = FmhaBwdCfg<D>;
  auto kern = fmha_bwd_kernel<D, DROP>;
  OFB_CUDA_OK_ONCE_PER_DEVICE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  p.n_kt = (p.Sk + 127) / 128;
  // heads walked together: as many as keep queries, gradients (bf16) and dQ (fp32) within a third of the L2 cache, but at
  // least one CTA for every SM
  const long long bh = static_cast<long long>(p.B) * p.Hk;
  long long chunk = (40ll << 20) / (static_cast<long long>(p.Sq) * D * 8 * (p.H / p.Hk));
  if (chunk * p.n_kt < 148) chunk = (148 + p.n_kt - 1) / p.n_kt;
  p.chunk = static_cast<int>(chunk < bh ? chunk : bh);
  const long long ctas = bh * p.n_kt;
  if (ctas > 0x7FFFFFFFll) return fail("fmha_bwd: too many key tiles");
  kern<<<static_cast<unsigned>(ctas), 512, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, tdq, p);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace ofb

using namespace ofb;

// Floats of scratch the backward needs: B*Sq*H*D for the fp32 dQ accumulator + B*H*Sq for delta.
OFB_API long long ofb_fmha_bwd_scratch_floats(int B, int S, int H, int D) {
  return static_cast<long long>(B) * S * H * D + static_cast<long long>(B) * H * S;
}

// q: [B,Sq,H,D] view (token stride q_row_stride); k, v: [B,Sk,Hk,D] views (kv_row_stride); o, d_o: contiguous
// [B,Sq,H,D]; dq: [B,Sq,H,D] view with token stride dq_row_stride; dk, dv: [B,Sk,Hk,D] views with token stride
// dkv_row_stride. scratch: ofb_fmha_bwd_scratch_floats(B, Sq, H, D) floats. Dropout arguments as in the forward call
// whose output is differentiated.
OFB_API int ofb_fmha_bwd_ex(const void* q, const void* k, const void* v, long long q_row_stride, long long kv_row_stride,
                            const void* o, const void* d_o, const float* lse, void* dq, void* dk, void* dv,
                            long long dq_row_stride, long long dkv_row_stride, float* scratch, const int* kv_len, int B,
                            int Sq, int Sk, int H, int Hk, int D, int causal, float scale, float p_dropout,
                            unsigned long long seed, unsigned int offset, void* stream) {
  if (D != 64 && D != 128) return fail("fmha_bwd: head dim must be 64 or 128");
  if (Hk <= 0 || H % Hk) return fail("fmha_bwd: the number of query heads must be a multiple of the key/value heads");
  if (dq_row_stride % 8 || dkv_row_stride % 8) return fail("fmha_bwd: gradient row strides must be multiples of 8");
  if (B <= 0 || Sq <= 0 || Sk <= 0) return fail("fmha_bwd: empty problem");
  auto s = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap tq, tk, tv, tdo;
  if (fmha_tensor_map(&tq, q, B, Sq, H, D, q_row_stride)) return -1;
  if (fmha_tensor_map(&tk, k, B, Sk, Hk, D, kv_row_stride)) return -1;
  if (fmha_tensor_map(&tv, v, B, Sk, Hk, D, kv_row_stride)) return -1;
  if (fmha_tensor_map(&tdo, d_o, B, Sq, H, D, static_cast<long long>(H) * D)) return -1;
  const long long n_acc = static_cast<long long>(B) * Sq * H * D;
  float* dq_acc = scratch;
  float* delta = scratch + n_acc;
  {
    const long long rows = static_cast<long long>(B) * Sq * H;
    const long long blocks = (rows * (D / 8) + 255) / 256;
    const __nv_bfloat16* po = reinterpret_cast<const __nv_bfloat16*>(o);
    const __nv_bfloat16* pd = reinterpret_cast<const __nv_bfloat16*>(d_o);
    if (D == 64) fmha_delta_kernel<64><<<static_cast<unsigned>(blocks), 256, 0, s>>>(po, pd, delta, dq_acc, B, Sq, H);
    else fmha_delta_kernel<128><<<static_cast<unsigned>(blocks), 256, 0, s>>>(po, pd, delta, dq_acc, B, Sq, H);
    OFB_CUDA_OK(cudaGetLastError());
  }
  FmhaBwdParams p;
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc;
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk); p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.dkv_row_stride = dkv_row_stride; p.kv_len = kv_len;
  p.B = B; p.H = H; p.Hk = Hk; p.Sq = Sq; p.Sk = Sk; p.D = D; p.causal = causal; p.causal_off = Sk - Sq;
  p.scale = scale; p.scale_log2e = scale * 1.4426950408889634f;
  p.status = device_status_ptr();
  if (fmha_dropout_cfg(&p.drop, p_dropout, seed, offset)) return -1;
  CUtensorMap tdq;
  {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return fail("cuTensorMapEncodeTiled is not available");
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)Sq, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)D * 4, (cuuint64_t)H * D * 4, (cuuint64_t)Sq * H * D * 4};
    cuuint32_t box[4] = {32, 1, 32, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dq_acc, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail("fmha_bwd: cuTensorMapEncodeTiled(dq) failed with code " + std::to_string((int)r));
  }
  int rc;
  if (p_dropout > 0.f)
    rc = D == 64 ? launch_fmha_bwd<64, true>(tq, tk, tv, tdo, tdq, p, s) : launch_fmha_bwd<128, true>(tq, tk, tv, tdo, tdq, p, s);
  else
    rc = D == 64 ? launch_fmha_bwd<64, false>(tq, tk, tv, tdo, tdq, p, s) : launch_fmha_bwd<128, false>(tq, tk, tv, tdo, tdq, p, s);
  if (rc) return rc;
  {
    const long long rows = static_cast<long long>(B) * Sq;
    const long long total = rows * (H * D / 8);
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    fmha_dq_cast_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(dq_acc, reinterpret_cast<__nv_bfloat16*>(dq), rows,
                                                                     H * D, dq_row_stride, scale);
    OFB_CUDA_OK(cudaGetLastError());
  }
  return 0;
}

// Self-attention form: one length, one head count, dq / dk / dv slices of one packed buffer.
OFB_API int ofb_fmha_bwd(const void* q, const void* k, const void* v, long long q_row_stride, long long kv_row_stride,
                         const void* o, const void* d_o, const float* lse, void* dq, void* dk, void* dv,
                         long long dqkv_row_stride, float* scratch, const int* kv_len, int B, int S, int H, int D,
                         int causal, float scale, void* stream) {
  return ofb_fmha_bwd_ex(q, k, v, q_row_stride, kv_row_stride, o, d_o, lse, dq, dk, dv, dqkv_row_stride, dqkv_row_stride, scratch,
                         kv_len, B, S, S, H, H, D, causal, scale, 0.f, 0ull, 0u, stream);
}
