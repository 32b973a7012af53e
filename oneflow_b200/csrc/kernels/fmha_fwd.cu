// Fused multi-head attention forward for sm_100a (bf16, head dim 64 or 128, causal or
// full, optional per-batch key length for padding, query length != key length with the causal
// diagonal aligned to the bottom-right corner, grouped-query attention: H query heads share
// Hk key/value heads, dropout on the probabilities from a Philox counter indexed by position).
//
// One CTA runs two independent softmax streams of 128 query rows against the same tensor core, so that the products of one
// stream hide behind the exponentials of the other. Roles:
//   warp 0      TMA producer: the query tile(s) once, then K / V tiles through a ring in the order the products use them
//   warp 1      tcgen05 issuer: S_t = Q_t K^T, then O_t += P_t V with P_t read from TMEM (it lies over the S_t it came from)
//   warps 4..7  softmax of stream 0, warps 8..11 of stream 1: one thread owns one whole query row (a TMEM lane), so row
//               maxima and sums need no exchange, and P goes back to TMEM without touching shared memory
// The streams are two neighbouring query tiles (kPairs: every K / V tile is loaded once for 256 rows), or, when that would leave
// SMs without a CTA, the even and the odd key tiles of ONE query tile whose two results are merged at the end (kSplit: twice the
// CTAs, half the chain), or the two halves of its only key tile (kOneTile). With dropout the random numbers are most of a stream's
// work: the last of an odd number of split tiles is halved too. (Without, the branches for that cost more than they gain: 128
// heads, 1 x 512, D = 128 10.7 against 10.1 us.)
//
// What bounds it: the exponentials (16 per clock and SM: 1024 clocks for a 128 x 128 tile) and the two products of a D = 128
// tile (1024 clocks) alike. Measured on a B200, forward alone, against a kernel of one stream (P through shared
// memory, two threads a row that meet at a barrier on every tile), and in brackets with one CTA per pair: batch 4, 32 heads,
// 2048 x 2048, D = 128, causal 283 -> 163 us (187); batch 1, 32 / 8 heads, 8192 x 8192, D = 128, causal 847 -> 451 us (470);
// batch 32, 16 heads, 512 x 512, D = 64 143 -> 73 us (88).
// Pairs: a running CTA takes over the next item that has not started (cluster launch control), so that the first loads of an
// item run under the end of the one before.
// The exponent reference trails the true running maximum by up to 2^8, so O is only rescaled in TMEM (tcgen05.ld / st) on
// the rare tiles where a row maximum jumps. tcgen05 products of one thread run in issue order, hence: S_t of the next tile
// is issued right behind the P_t V that reads the same columns, and a finished S_t means that the P V before it is finished.
//
// Reference counterparts: oneflow/user/kernels/scaled_dot_product_attention_kernel.cu (flash
// attention library call), fused_attention_kernels.cu :710 (CUTLASS fMHA, no sm_100 path) and the
// unfused fused_tril_scale_softmax_mask_scale chain.
#include "../common/host_utils.h"
#include "../common/philox.cuh"
#include "../common/ptx.cuh"
#include "ofb_kernels.h"

namespace ofb {

struct FmhaFwdParams {
  __nv_bfloat16* out;   // [B, Sq, H, D] contiguous
  float* lse;           // [B, H, Sq] natural-log sum-exp of the scaled scores
  const int* kv_len;    // [B] number of valid keys per batch or null
  int B, H, Hk, Sq, Sk, D;   // H query heads, Hk key/value heads (H % Hk == 0)
  int causal;
  int causal_off;       // Sk - Sq: query row r sees key columns <= r + causal_off
  DropoutCfg drop;
  float scale_log2e;    // softmax scale * log2(e)
  int n_qt;             // query tiles (SPLIT) or pairs of query tiles of one head
  int chunk;            // heads (of B * H) that are walked together, longest tiles first
  int* status;
};

template <int D>
struct FmhaFwdCfg {
  static constexpr int BM = 128, BN = 128;
  static constexpr int Q_BYTES = BM * D * 2;            // one query tile
  static constexpr int KV_BYTES = BN * D * 2;
  static constexpr int SLOTS = D == 128 ? 5 : 8;        // K / V ring
  static constexpr int BAR_BYTES = 320;                 // mbarriers, the TMEM slot, the abort flag, two answers of 16 bytes
  static constexpr int XCHG_BYTES = 2 * 128 * 8;        // SPLIT: row maximum and sum of both streams
  // At D = 128 the tiles take 224 KiB of the 227 KiB a CTA may have: the dynamic shared memory is declared 1024-byte
  // aligned (the kernel has no static shared memory, so it starts the CTA's window) instead of being aligned by hand
  // with a kilobyte of slack; the kernel checks the alignment and reports a status instead of running if it is not there.
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + SLOTS * KV_BYTES + BAR_BYTES + XCHG_BYTES;
};

// How the two streams of a CTA share the work.
enum FmhaFwdMode {
  kPairs = 0,      // two neighbouring query tiles
  kSplit = 1,      // the even and the odd key tiles of one query tile
  kOneTile = 2,    // no more than 128 keys: their first and second 64
};

template <int D, bool DROP, int MODE>
__global__ void __launch_bounds__(384, 1)
fmha_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, FmhaFwdParams p) {
  using Cfg = FmhaFwdCfg<D>;
  constexpr int BM = 128, BN = 128, DCH = D / 64;  // 64-element chunks along the head dimension
  constexpr int SLOTS = Cfg::SLOTS;
  constexpr bool SPLIT = MODE != kPairs, ONE = MODE == kOneTile;
  constexpr bool HALVE = ONE || (SPLIT && DROP);   // whether a key tile may be shared by the streams, 64 keys each
  constexpr uint32_t IDESC_S = make_idesc_bf16(BM, BN, 0, 0), IDESC_S_HALF = make_idesc_bf16(BM, BN / 2, 0, 0);
  constexpr uint32_t IDESC_O = make_idesc_bf16(BM, D, 0, 1);
  constexpr int CH_BYTES = 128 * 128;  // one [128 rows x 64 elements] swizzled chunk

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {   // uniform over the CTA: nobody has touched a barrier or TMEM yet
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, (int)kStatusBounds);
    return;
  }
  uint8_t* sQ = smem;                         // 2 tiles
  uint8_t* sKV = sQ + 2 * Cfg::Q_BYTES;       // ring of K and V tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + SLOTS * Cfg::KV_BYTES);
  uint64_t* q_full = bars;               // [2]
  uint64_t* kv_full = bars + 2;          // [SLOTS]
  uint64_t* kv_empty = kv_full + SLOTS;  // [SLOTS]
  uint64_t* s_full = kv_empty + SLOTS;   // [2]
  uint64_t* p_full = s_full + 2;         // [2] 128 softmax threads of the stream
  uint64_t* o_done = p_full + 2;         // [2]
  uint64_t* pair_bar = o_done + 2;       // SPLIT: all 256 softmax threads, once
  uint64_t* q_empty = pair_bar + 1;      // every product of an item has finished
  uint64_t* o_free = q_empty + 1;        // [2] 128 softmax threads: O has left TMEM
  uint64_t* next_full = o_free + 2;      // [2] the answer that names the CTA's next item
  uint64_t* next_empty = next_full + 2;  // [2] 10 warps
  uint8_t* answers = reinterpret_cast<uint8_t*>(bars + 32);   // [2] 16 bytes
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(answers + 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert(2 + 2 * SLOTS + 7 + 7 <= 32 && 32 * 8 + 32 + 8 <= Cfg::BAR_BYTES, "barriers do not fit");
  float2* xchg = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(bars) + Cfg::BAR_BYTES);   // [2 streams][128 rows]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Item `n` of the grid: CTAs walk the heads in chunks whose keys and values stay in L2 together; inside a chunk the longest
  // (last) causal tiles of all its heads come first, so that the short ones fill the tail.
  struct Item {
    int q0, bh, h, b, hk, kv_limit;
    int n_it[2];     // key tiles of each stream
    bool shared;     // HALVE: both streams take half of the last tile
  };
  auto item_of = [&](int item) {
    const int in_chunk_max = p.chunk * p.n_qt;
    const int ck = item / in_chunk_max, rem = item % in_chunk_max;
    const int heads_here = min(p.chunk, p.B * p.H - ck * p.chunk);
    Item it;
    it.q0 = (p.n_qt - 1 - rem / heads_here) * (SPLIT ? BM : 2 * BM);
    it.bh = ck * p.chunk + rem % heads_here;
    it.h = it.bh % p.H;
    it.b = it.bh / p.H;
    it.hk = it.h / (p.H / p.Hk);
    it.kv_limit = p.kv_len ? min(p.Sk, p.kv_len[it.b]) : p.Sk;
    // all key tiles that a stream's rows see, or every second one of them. Rows grow with the stream, so stream 1 never sees
    // fewer tiles than stream 0 unless it has no rows at all.
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int r0 = SPLIT ? it.q0 : it.q0 + t * BM;
      int kv_end = it.kv_limit;
      if (p.causal) kv_end = min(kv_end, r0 + BM + p.causal_off);
      const int n = (kv_end > 0 && r0 < p.Sq) ? (kv_end + BN - 1) / BN : 0;
      it.shared = HALVE && (n & 1) && kv_end - (n - 1) * BN > BN / 2;    // its second half holds a key that some row sees
      it.n_it[t] = SPLIT ? (n + (t == 0 || it.shared)) >> 1 : n;
    }
    return it;
  };
  // Pairs: the CTA works through items until none is left, every role walks the same sequence (`n` counts them). Split key tiles
  // come in one wave or two: one item per CTA.
  auto next_item = [&](int n, int& item) -> bool {      // called by whole warps
    if constexpr (SPLIT) {
      return false;
    } else {
      const bool ok = mbar_wait(&next_full[n & 1], (n >> 1) & 1, abort_flag);
      int nx = 0;
      const bool more = ok && clc_take(answers + (n & 1) * 16, nx);
      item = nx;
      __syncwarp();
      if (lane == 0) mbar_arrive(&next_empty[n & 1]);
      return more;
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 128);
      mbar_init(&o_done[t], 1);
    }
    mbar_init(pair_bar, 256);
    mbar_init(q_empty, 1);
    for (int t = 0; t < 2; ++t) {
      mbar_init(&o_free[t], 128);
      mbar_init(&next_full[t], 1);
      mbar_init(&next_empty[t], 10);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base;            // S[0], S[1] at +0, +128; P[t] takes the first 64 columns of S[t]
  const uint32_t tO = tmem_base + 256;      // O[0], O[1] at +0, +128, D columns each

  // registers: 384 threads x 168 at launch = 3 warpgroups x (88 + 208 + 208); a softmax thread holds a whole row of S. (With 72
  // for the producer and issuer their few spills cost 10 %: 181 instead of 163 us at batch 4, 32 heads, 2048 x 2048, causal.)
  if (warp < 4) {
    reg_dec<88>();
    if (warp == 0) {
      int item = blockIdx.x;
      int c = 0;                             // loads issued so far: load c uses slot c % SLOTS
      int act = 0;                           // items before this one that had any key tile
      bool ok = true;
      for (int n = 0;; ++n) {
        const Item it = item_of(item);
        const int tiles = ONE ? it.n_it[0] : SPLIT ? it.n_it[0] + it.n_it[1] - it.shared : max(it.n_it[0], it.n_it[1]);
        if (elect_one()) {
          auto load_kv = [&](const CUtensorMap* m, int tile) -> bool {
            const int s = c % SLOTS;
            if (!mbar_wait(&kv_empty[s], ((c / SLOTS) & 1) ^ 1, abort_flag)) return false;
            mbar_arrive_expect_tx(&kv_full[s], Cfg::KV_BYTES);
#pragma unroll
            for (int d = 0; d < DCH; ++d)
              tma_load_4d(sKV + s * Cfg::KV_BYTES + d * CH_BYTES, m, &kv_full[s], d * 64, it.hk, tile * BN, it.b);
            ++c;
            return true;
          };
          auto load_q = [&](int t) {      // only what a product will wait for: no copy may be in flight when the CTA leaves
            if (it.n_it[t] == 0) return;
            mbar_arrive_expect_tx(&q_full[t], Cfg::Q_BYTES);
#pragma unroll
            for (int d = 0; d < DCH; ++d)
              tma_load_4d(sQ + t * Cfg::Q_BYTES + d * CH_BYTES, &tmQ, &q_full[t], d * 64, it.h, it.q0 + t * BM, it.b);
          };
          // a few tiles before the loads of this item end (see the backward kernel)
          auto ask = [&]() {
            if (!mbar_wait(&next_empty[n & 1], ((n >> 1) & 1) ^ 1, abort_flag)) return;
            fence_proxy_async_smem();
            clc_ask(answers + (n & 1) * 16, &next_full[n & 1]);
          };
          if constexpr (SPLIT) {
            if (tiles > 0) {
              load_q(0);
              ok = load_kv(&tmK, 0);
              if (tiles > 1) ok = ok && load_kv(&tmK, 1);
              for (int g = 0; g < tiles && ok; ++g) {
                ok = load_kv(&tmV, g);
                if (ok && g + 2 < tiles) ok = load_kv(&tmK, g + 2);
              }
            }
          } else {
            const int ask_at = max(0, tiles - 4);
            if (tiles == 0 || !ok) ask();
            if (tiles > 0 && ok) {
              ok = load_kv(&tmK, 0) && mbar_wait(q_empty, (act & 1) ^ 1, abort_flag);
              if (ok) {
                load_q(0);
                load_q(1);
              }
              for (int i = 0; i < tiles; ++i) {
                if (i == ask_at) ask();
                ok = ok && load_kv(&tmV, i);
                if (ok && i + 1 < tiles) ok = load_kv(&tmK, i + 1);
              }
            }
          }
        }
        __syncwarp();
        act += tiles > 0;
        if (!next_item(n, item)) break;
      }
    } else if (warp == 1) {
      int item = blockIdx.x;
      int c0 = 0;                            // loads of the items before this one
      int act = 0;
      int j0[2] = {0, 0}, seen[2] = {0, 0};  // key tiles and items each stream had before this item
      bool ok = true;
      for (int n = 0;; ++n) {
        const Item it = item_of(item);
        const int tiles = ONE ? it.n_it[0] : SPLIT ? it.n_it[0] + it.n_it[1] - it.shared : max(it.n_it[0], it.n_it[1]);
        if (elect_one() && tiles > 0 && ok) {
          const uint32_t kv_base = smem_u32(sKV);
          auto slot_ready = [&](int c) -> bool { return mbar_wait(&kv_full[c % SLOTS], (c / SLOTS) & 1, abort_flag); };
          // S_t = Q_t K^T with the K tile of load c, or (half) with its keys 64 t .. 64 t + 63: eight groups of eight rows further
          auto issue_s = [&](int t, int c, bool half) {
            const uint32_t q_base = smem_u32(sQ + (SPLIT ? 0 : t) * Cfg::Q_BYTES);
            const uint32_t k_base = kv_base + (c % SLOTS) * Cfg::KV_BYTES + (half ? t * 8192 : 0);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const uint32_t off = (kk >> 2) * CH_BYTES + (kk & 3) * 32;
              umma_bf16_ss(tS + t * BN, make_smem_desc_sw128(q_base + off, 16, 1024), make_smem_desc_sw128(k_base + off, 16, 1024),
                           half ? IDESC_S_HALF : IDESC_S, kk != 0 ? 1u : 0u);
            }
            umma_commit(&s_full[t]);
          };
          auto issue_pv = [&](int t, int c, bool first, bool half) {   // O_t (+)= P_t V with the V tile of load c, or with its half
            const uint32_t v_base = kv_base + (c % SLOTS) * Cfg::KV_BYTES + (half ? t * 8192 : 0);
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk)
              if (kk < BN / 32 || !half)
                umma_bf16_ts(tO + t * 128, tS + t * BN + kk * 8, make_smem_desc_sw128(v_base + kk * 2048, CH_BYTES, 1024), IDESC_O,
                             (first && kk == 0) ? 0u : 1u);
          };
          auto release = [&](int c) { umma_commit(&kv_empty[c % SLOTS]); };
          if constexpr (SPLIT) {
            // loads come in the order K0 K1 V0 K2 V1 K3 ... of the producer; a shared tile's stay until stream 1 has used them too
            // (for good where there is only one)
            auto halved = [&](int g) { return ONE || (HALVE && it.shared && g == tiles - 1); };
            auto next_s = [&](int t, int g) -> bool {
              const int c = g == 0 ? 0 : 2 * g - 1;
              if (!slot_ready(c)) return false;
              tc_fence_after();
              issue_s(t, c, halved(g));
              if (!ONE && (!halved(g) || t == 1)) release(c);
              return true;
            };
            auto next_pv = [&](int t, int g) -> bool {
              const int c = g == tiles - 1 ? 2 * tiles - 1 : 2 * g + 2;
              if (!mbar_wait(&p_full[t], (g >> 1) & 1, abort_flag) || !slot_ready(c)) return false;
              tc_fence_after();
              issue_pv(t, c, g < 2, halved(g));
              if (!ONE && (!halved(g) || t == 1)) release(c);
              return true;
            };
            ok = mbar_wait(&q_full[0], 0, abort_flag) && next_s(0, 0);
            if (!ONE && tiles > 1) ok = ok && next_s(1, 1);
            else if (it.shared) ok = ok && next_s(1, 0);
            for (int g = 0; g < tiles && ok; ++g) {
              if (halved(g)) {
                ok = next_pv(0, g);
                if (ok) umma_commit(&o_done[0]);
                if (it.shared) {
                  ok = ok && next_pv(1, g);
                  if (ok) umma_commit(&o_done[1]);
                }
              } else {
                const int t = g & 1;
                ok = next_pv(t, g);
                if (!ok) break;
                if (g + 2 < tiles) ok = next_s(t, g + 2);
                else if (HALVE && t == 1 && it.shared) ok = next_s(1, tiles - 1);
                else umma_commit(&o_done[t]);
              }
            }
          } else {
            ok = slot_ready(c0);
            for (int t = 0; t < 2 && ok; ++t) {
              if (it.n_it[t] == 0) continue;
              ok = mbar_wait(&q_full[t], seen[t] & 1, abort_flag);
              if (!ok) break;
              tc_fence_after();
              issue_s(t, c0, false);
            }
            if (ok) release(c0);
            for (int i = 0; i < tiles && ok; ++i) {
              const int cv = c0 + 2 * i + 1, ck1 = c0 + 2 * i + 2;      // loads of V_i and K_{i+1}
              for (int t = 0; t < 2; ++t) {
                if (i >= it.n_it[t]) continue;
                if (!mbar_wait(&p_full[t], (j0[t] + i) & 1, abort_flag) || !slot_ready(cv)) { ok = false; break; }
                // O of the item before has left TMEM
                if (i == 0 && !mbar_wait(&o_free[t], (seen[t] & 1) ^ 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                issue_pv(t, cv, i == 0, false);
                if (t == 1 || i >= it.n_it[1]) release(cv);       // the last stream to use the tile
                if (i + 1 < it.n_it[t]) {
                  if (!slot_ready(ck1)) { ok = false; break; }
                  tc_fence_after();
                  issue_s(t, ck1, false);
                  if (t == 1 || i + 1 >= it.n_it[1]) release(ck1);
                } else {
                  umma_commit(&o_done[t]);
                }
              }
            }
            if (ok) umma_commit(q_empty);
          }
        }
        __syncwarp();
        c0 += 2 * tiles;
        act += tiles > 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          j0[t] += it.n_it[t];
          seen[t] += it.n_it[t] > 0;
        }
        if (!next_item(n, item)) break;
      }
    }
  } else {
    reg_inc<208>();
    const int quad = warp & 3;
    const int t = (warp - 4) >> 2;           // stream
    const int r = quad * 32 + lane;          // row inside the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tSt = tS + lane_addr + t * BN, tOt = tO + lane_addr + t * 128;
    int item = blockIdx.x;
    int j0 = 0, seen = 0;                    // key tiles and items this stream had before this item
    bool ok = true;
    for (int n = 0;; ++n) {
      const Item it = item_of(item);
      const int row0 = SPLIT ? it.q0 : it.q0 + t * BM;
      const int row_g = row0 + r;
      const int nt = it.n_it[t];
      // m_ref is the exponent reference actually used for P and l; it trails the true running maximum by at
      // most kLazy (log2 units) so that the TMEM-resident O only has to be rescaled when the maximum jumps.
      constexpr float kLazy = 8.0f;
      float m_ref = -INFINITY, l_run = 0.f;
      const uint64_t scale2 = pack_f32x2(__float_as_uint(p.scale_log2e), __float_as_uint(p.scale_log2e));
      const int col_max = p.causal ? min(row_g + p.causal_off, it.kv_limit - 1) : it.kv_limit - 1;  // last visible column
      for (int i = 0; i < nt && ok && (!ONE || i == 0); ++i) {
        const bool half = ONE || (HALVE && it.shared && i == nt - 1);
        const int col_base = half ? 2 * i * BN + t * (BN / 2) : (SPLIT ? 2 * i + t : i) * BN;
        const int nc = half ? 2 : 4, width = nc * 32;      // chunks of 32 key columns
        if (!mbar_wait(&s_full[t], (j0 + i) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const bool need_mask = (p.causal && col_base + width - 1 > row0 + p.causal_off) || (col_base + width > it.kv_limit);
        uint32_t sv[4][32];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c < nc) {
            tmem_ld_32x32(tSt + c * 32, sv[c]);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[c][e] = 0xFF800000u;
          }
        }
        tmem_wait_ld();
        if (need_mask) {
          const int lim = col_max - col_base;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e > lim) sv[c][e] = 0xFF800000u;   // -inf
        }
        // the scores stay unscaled here: the scale is positive, so the maximum commutes with it, and the exponent below
        // applies it inside one fused multiply-add. Eight chains: a dependent chain of 128 cannot be hidden.
        float mxs[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) mxs[e] = fmaxf(__uint_as_float(sv[0][e]), __uint_as_float(sv[0][e + 8]));
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = (c == 0 ? 16 : 0); e < 32; e += 16)
#pragma unroll
            for (int k = 0; k < 8; ++k)
              mxs[k] = fmaxf(fmaxf(mxs[k], __uint_as_float(sv[c][e + k])), __uint_as_float(sv[c][e + 8 + k]));
        float mx = fmaxf(fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])), fmaxf(fmaxf(mxs[4], mxs[5]), fmaxf(mxs[6], mxs[7])));
        mx *= p.scale_log2e;   // -inf stays -inf
        // Rescale O (and l) only when some row of the warp moved its maximum by more than kLazy. S of this tile is finished,
        // so every product of the tiles before it is: O may be touched without another wait.
        if (__any_sync(0xffffffffu, mx > m_ref + kLazy)) {
          const float m_new = fmaxf(m_ref, mx);
          const float alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - m_new);  // m_new is finite here or equals m_ref
          if (!ONE && i > 0) {
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) {
              uint32_t o[16];
              tmem_ld_32x16(tOt + cc * 16, o);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st_32x16(tOt + cc * 16, o);
            }
          }
          l_run *= alpha;
          m_ref = m_new;
        }
        const float m_neg = m_ref == -INFINITY ? 0.f : -m_ref;
        const uint64_t m_neg2 = pack_f32x2(__float_as_uint(m_neg), __float_as_uint(m_neg));
        uint64_t rs[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= nc) continue;
          uint32_t packed[16];
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            float pv[4];
            unpack_f32x2(fma_f32x2(pack_f32x2(sv[c][e], sv[c][e + 1]), scale2, m_neg2), pv[0], pv[1]);
            unpack_f32x2(fma_f32x2(pack_f32x2(sv[c][e + 2], sv[c][e + 3]), scale2, m_neg2), pv[2], pv[3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) pv[k] = fast_exp2(pv[k]);   // masked entries are -inf -> 0
            rs[(e >> 1) & 3] = add_f32x2(rs[(e >> 1) & 3], pack_f32x2(__float_as_uint(pv[0]), __float_as_uint(pv[1])));
            rs[((e >> 1) + 1) & 3] = add_f32x2(rs[((e >> 1) + 1) & 3], pack_f32x2(__float_as_uint(pv[2]), __float_as_uint(pv[3])));
            if constexpr (DROP) {
              // the row sum keeps every probability; only what multiplies V is dropped (1 / keep is applied at the end)
              const uint32_t keep = dropout_keep4(p.drop, static_cast<uint32_t>(it.bh), static_cast<uint32_t>(row_g),
                                                  static_cast<uint32_t>((col_base + c * 32 + e) >> 2));
#pragma unroll
              for (int k = 0; k < 4; ++k) pv[k] = (keep >> k) & 1u ? pv[k] : 0.f;
            }
            packed[e >> 1] = pack_bf16x2(pv[0], pv[1]);
            packed[(e >> 1) + 1] = pack_bf16x2(pv[2], pv[3]);
          }
          tmem_st_32x16(tSt + c * 16, packed);    // the whole row of S has left TMEM above
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(&p_full[t]);
        float lo, hi;
        unpack_f32x2(add_f32x2(add_f32x2(rs[0], rs[1]), add_f32x2(rs[2], rs[3])), lo, hi);
        l_run += lo + hi;
      }
      if (ok && nt > 0) ok = mbar_wait(&o_done[t], seen & 1, abort_flag);
      __nv_bfloat16* orow = p.out + ((static_cast<long long>(it.b) * p.Sq + row_g) * p.H + it.h) * D;
      float* lse = p.lse ? p.lse + (static_cast<long long>(it.b) * p.H + it.h) * p.Sq + row_g : nullptr;
      if constexpr (SPLIT) {
        // O = (2^(m0 - m) O_0 + 2^(m1 - m) O_1) / l: both streams' accumulators lie in the same TMEM lanes, so each stream's
        // threads write one half of the columns of the merged row.
        if (ok) {
          xchg[t * 128 + r] = make_float2(m_ref, l_run);
          tc_fence_before();
          mbar_arrive(pair_bar);
          ok = mbar_wait(pair_bar, 0, abort_flag);
        }
        if (ok) {
          tc_fence_after();
          const float2 other = xchg[(t ^ 1) * 128 + r];
          const float m0 = t == 0 ? m_ref : other.x, m1 = t == 0 ? other.x : m_ref;
          const float l0 = t == 0 ? l_run : other.y, l1 = t == 0 ? other.y : l_run;
          const float m = fmaxf(m0, m1);
          const float a0 = m0 == -INFINITY ? 0.f : exp2f(m0 - m), a1 = m1 == -INFINITY ? 0.f : exp2f(m1 - m);
          const float l_tot = a0 * l0 + a1 * l1;
          const float inv = l_tot > 0.f ? (DROP ? p.drop.inv_keep : 1.f) / l_tot : 0.f;
          const float w0 = a0 * inv, w1 = a1 * inv;
#pragma unroll
          for (int c0 = 0; c0 < D / 64; ++c0) {
            const int cc = t * (D / 64) + c0;
            uint32_t u[32], v[32];
            __syncwarp();
            // an accumulator that no product wrote holds whatever TMEM held before: it must not enter the sum even with weight 0
            if (it.n_it[0] > 0) tmem_ld_32x32(tO + lane_addr + cc * 32, u);
            if (it.n_it[1] > 0) tmem_ld_32x32(tO + lane_addr + 128 + cc * 32, v);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              float f = it.n_it[0] > 0 ? __uint_as_float(u[e]) * w0 : 0.f;
              if (it.n_it[1] > 0) f = fmaf(__uint_as_float(v[e]), w1, f);
              u[e] = __float_as_uint(f);
            }
            if (row_g < p.Sq) {
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                uint32_t w4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w4[e] = pack_bf16x2(__uint_as_float(u[g * 8 + 2 * e]), __uint_as_float(u[g * 8 + 2 * e + 1]));
                *reinterpret_cast<uint4*>(orow + cc * 32 + g * 8) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
              }
            }
          }
          if (t == 0 && row_g < p.Sq && lse) *lse = l_tot > 0.f ? (m + log2f(l_tot)) * 0.6931471805599453f : -INFINITY;
        }
      } else if (ok && nt > 0) {
        tc_fence_after();
        const float inv = l_run > 0.f ? (DROP ? p.drop.inv_keep : 1.f) / l_run : 0.f;
#pragma unroll
        for (int cc = 0; cc < D / 32; ++cc) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(tOt + cc * 32, v);
          tmem_wait_ld();
          if (row_g < p.Sq) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[g * 8 + e]) * inv;
              *reinterpret_cast<uint4*>(orow + cc * 32 + g * 8) =
                  make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&o_free[t]);
        if (row_g < p.Sq && lse) *lse = l_run > 0.f ? (m_ref + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
      } else if (ok && row_g < p.Sq) {
        // No visible keys at all (kv_len == 0, or a causal tile above the shifted diagonal): the output rows are zero.
        for (int e = 0; e < D; e += 8) *reinterpret_cast<uint4*>(orow + e) = make_uint4(0, 0, 0, 0);
        if (lse) *lse = -INFINITY;
      }
      j0 += nt;
      seen += nt > 0;
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

template <int D, bool DROP, int MODE>
static int launch_fmha_fwd_as(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, FmhaFwdParams p,
                              cudaStream_t stream) {
  using Cfg = FmhaFwdCfg<D>;
  auto kern = fmha_fwd_kernel<D, DROP, MODE>;
  OFB_CUDA_OK_ONCE_PER_DEVICE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  p.n_qt = MODE == kPairs ? (p.Sq + 255) / 256 : (p.Sq + 127) / 128;
  // heads walked together: as many as keep their keys and values within a third of the L2 cache (the query heads of a group
  // share theirs), but at least one CTA for every SM
  const long long bh = static_cast<long long>(p.B) * p.H;
  long long chunk = (40ll << 20) / (static_cast<long long>(p.Sk) * D * 4) * (p.H / p.Hk);
  if (chunk * p.n_qt < 148) chunk = (148 + p.n_qt - 1) / p.n_qt;
  p.chunk = static_cast<int>(chunk < bh ? chunk : bh);
  const long long ctas = bh * p.n_qt;
  if (ctas > 0x7FFFFFFFll) return fail("fmha: too many query tiles");
  kern<<<static_cast<unsigned>(ctas), 384, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, p);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int D, bool DROP>
static int launch_fmha_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FmhaFwdParams& p,
                           cudaStream_t stream) {
  const long long bh = static_cast<long long>(p.B) * p.H;
  const long long pairs = bh * ((p.Sq + 255) / 256), tiles = bh * ((p.Sq + 127) / 128);
  // Up to 128 keys a CTA's whole work is one tile: halved between the streams, by a kernel without ring, loop and rescaling, it takes 4.7 us
  // instead of 5.8 (8 heads, 1 x 64, D = 64; with dropout 5.9 and 8.6). Pairs do not start a CTA per tile, which pays from two
  // tiles an SM on (1024 heads, 64 x 64: 27 against 29 us), but not while a second wave of them does one tile of two (96 heads,
  // 300 x 100: 10.7 against 12.6 us). With dropout the random numbers are most of the work, and halves of tiles balance it best
  // (1024 heads, 64 x 64: 38 against 49 us; 128 x 128: 45 against 48).
  if (p.Sk <= 128) {
    if (DROP || tiles <= 148 || (p.Sq > 128 && pairs > 148 && tiles <= 2 * 148))
      return launch_fmha_fwd_as<D, DROP, kOneTile>(tq, tk, tv, p, stream);
    return launch_fmha_fwd_as<D, DROP, kPairs>(tq, tk, tv, p, stream);
  }
  // Pairs of query tiles load every key once for 256 rows, but give half the CTAs of split key tiles, each with twice the
  // chain. Splitting pays while all its CTAs run at once (batch 1, 8 heads, 2048 keys, D = 64: 20.3 against 33.9 us), and under
  // a causal mask also up to one wave of pairs, as the short tiles of the second wave fill in behind the long ones (16 heads,
  // 2048 keys, D = 128: 29.3 against 37.9 us; 4 heads, 8192 keys: 67 against 125 us) once there are keys enough to split
  // (64 heads, 512 keys: 19.1 against 16.3 us). Otherwise pairs win (16 heads, 2048 keys, D = 128, full: 38.7 against 44.5 us;
  // 16 heads, 4096 keys, causal: 71 against 82 us).
  bool split = tiles <= 148 || (p.causal && pairs < 148 && p.Sk >= 1024);
  if constexpr (DROP) {
    // The random numbers bind both forms to a time per step of a stream, so that waves of CTAs decide: a key tile takes a pair one
    // step of each stream and split tiles half a step; beside the steps a wave costs 0.6 and 0.75 of one. Measured: 80 heads, 494 x
    // 494, D = 64, causal 39 us in two waves of pairs, 30 us in three of split tiles; 24 heads, 3357 x 3357, D = 128 478 and
    // 381 us; 512 heads, 512 x 512, D = 64 174 and 208 us; 256 heads, 1 x 2048, D = 128 157 and 95 us.
    const long long nk = (p.Sk + 127) / 128, wp = (pairs + 147) / 148, wt = (tiles + 147) / 148;
    split = split || wt * (10 * nk + 15) < wp * (20 * nk + 12);
  } else {
    // With one query tile a head a pair has only one, whose stream walks all keys while the other has nothing to do: split from
    // five key tiles on (256 heads, 1 x 2048, D = 128: 49 against 62 us; 320 heads, 100 x 600: 35.6 against 37.4; but 640 heads,
    // 128 x 256, D = 64: 30 against 26, 2048 heads, 1 x 512, D = 128: 125 against 116).
    split = split || (p.Sq <= 128 && p.Sk > 512);
  }
  if (split) return launch_fmha_fwd_as<D, DROP, kSplit>(tq, tk, tv, p, stream);
  return launch_fmha_fwd_as<D, DROP, kPairs>(tq, tk, tv, p, stream);
}

// 4-D map over a [B, S, H, D] view with a token stride of `row_stride` elements.
int fmha_tensor_map(CUtensorMap* out, const void* ptr, int B, int S, int H, int D, long long row_stride) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail("cuTensorMapEncodeTiled is not available");
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (row_stride * 2) % 16) return fail("fmha: operands must be 16-byte aligned");
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)row_stride * 2, (cuuint64_t)row_stride * 2 * S};
  cuuint32_t box[4] = {64, 1, 128, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("fmha: cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return 0;
}

// Fills a DropoutCfg from a drop probability, a 64-bit seed and a per-call offset.
int fmha_dropout_cfg(DropoutCfg* d, float p_dropout, unsigned long long seed, unsigned int offset) {
  if (!(p_dropout >= 0.f) || p_dropout >= 1.f) return fail("fmha: dropout probability must be in [0, 1)");
  const double keep = 1.0 - static_cast<double>(p_dropout);
  const double t = keep * 4294967296.0;
  d->seed_lo = static_cast<uint32_t>(seed);
  d->seed_hi = static_cast<uint32_t>(seed >> 32);
  d->offset = offset;
  d->threshold = t >= 4294967295.0 ? 0xFFFFFFFFu : static_cast<uint32_t>(t);
  d->inv_keep = static_cast<float>(1.0 / keep);
  return 0;
}

__global__ void fmha_dropout_mask_kernel(DropoutCfg d, unsigned char* __restrict__ mask, int BH, int Sq, int Sk) {
  const long long groups = (Sk + 3) / 4;
  const long long total = static_cast<long long>(BH) * Sq * groups;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const uint32_t cg = static_cast<uint32_t>(i % groups);
    const uint32_t row = static_cast<uint32_t>((i / groups) % Sq);
    const uint32_t bh = static_cast<uint32_t>(i / (groups * Sq));
    const uint32_t keep = dropout_keep4(d, bh, row, cg);
    for (int e = 0; e < 4; ++e) {
      const long long col = 4ll * cg + e;
      if (col < Sk) mask[(static_cast<long long>(bh) * Sq + row) * Sk + col] = (keep >> e) & 1u;
    }
  }
}

}  // namespace ofb

using namespace ofb;

// q: bf16 view [B, Sq, H, D], element (b, s, h, d) at ((b*Sq + s) * q_row_stride + h*D + d); k, v: [B, Sk, Hk, D] views
// with token stride kv_row_stride. out: contiguous [B, Sq, H, D]; lse: [B, H, Sq]. With causal set, query row r sees
// key columns <= r + (Sk - Sq). p_dropout > 0 drops probabilities by the Philox stream (seed, offset).
OFB_API int ofb_fmha_fwd_ex(const void* q, const void* k, const void* v, long long q_row_stride, long long kv_row_stride,
                            void* out, float* lse, const int* kv_len, int B, int Sq, int Sk, int H, int Hk, int D, int causal,
                            float scale, float p_dropout, unsigned long long seed, unsigned int offset, void* stream) {
  if (D != 64 && D != 128) return fail("fmha: head dim must be 64 or 128");
  if (Hk <= 0 || H % Hk) return fail("fmha: the number of query heads must be a multiple of the key/value heads");
  if (B <= 0 || Sq <= 0 || Sk <= 0) return fail("fmha: empty problem");
  if (!(scale > 0.f)) return fail("fmha: the softmax scale must be positive");   // the kernel takes row maxima before scaling
  CUtensorMap tq, tk, tv;
  if (fmha_tensor_map(&tq, q, B, Sq, H, D, q_row_stride)) return -1;
  if (fmha_tensor_map(&tk, k, B, Sk, Hk, D, kv_row_stride)) return -1;
  if (fmha_tensor_map(&tv, v, B, Sk, Hk, D, kv_row_stride)) return -1;
  FmhaFwdParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse; p.kv_len = kv_len; p.B = B; p.H = H; p.Hk = Hk; p.Sq = Sq; p.Sk = Sk; p.D = D; p.causal = causal;
  p.causal_off = Sk - Sq;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.status = device_status_ptr();
  if (fmha_dropout_cfg(&p.drop, p_dropout, seed, offset)) return -1;
  auto s = reinterpret_cast<cudaStream_t>(stream);
  if (p_dropout > 0.f) return D == 64 ? launch_fmha_fwd<64, true>(tq, tk, tv, p, s) : launch_fmha_fwd<128, true>(tq, tk, tv, p, s);
  return D == 64 ? launch_fmha_fwd<64, false>(tq, tk, tv, p, s) : launch_fmha_fwd<128, false>(tq, tk, tv, p, s);
}

OFB_API int ofb_fmha_fwd(const void* q, const void* k, const void* v, long long q_row_stride, long long kv_row_stride,
                         void* out, float* lse, const int* kv_len, int B, int S, int H, int D, int causal, float scale,
                         void* stream) {
  return ofb_fmha_fwd_ex(q, k, v, q_row_stride, kv_row_stride, out, lse, kv_len, B, S, S, H, H, D, causal, scale, 0.f, 0ull, 0u,
                         stream);
}

// mask[b*H + h, row, col] = 1 where the attention dropout of (seed, offset) keeps the probability: the mask the fused
// kernels regenerate on the fly, written out for tests and for the unfused fallback.
OFB_API int ofb_fmha_dropout_mask(unsigned char* mask, int BH, int Sq, int Sk, float p_dropout, unsigned long long seed,
                                  unsigned int offset, void* stream) {
  DropoutCfg d;
  if (fmha_dropout_cfg(&d, p_dropout, seed, offset)) return -1;
  const long long total = static_cast<long long>(BH) * Sq * ((Sk + 3) / 4);
  if (total <= 0) return 0;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  fmha_dropout_mask_kernel<<<static_cast<unsigned>(blocks), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(d, mask, BH, Sq, Sk);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
