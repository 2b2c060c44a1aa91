// Forward attention for text queries on tcgen05 tensor cores: Kwai Summary
// Attention (sliding chunk window + old-chunk summaries), plain causal attention
// and token-sliding-window attention share this kernel.
//
// A work item is one tile of 128 query rows for TWO query heads of the same KV
// group ("slots"), so every K/V tile fetched by TMA feeds two S = Q K^T and two
// O += P V products and the two softmax warpgroups ping-pong against the tensor
// pipe.  Key tiles come from a closed-form range (attn_common.cuh): summary-key
// tiles first, then the text-key tiles of the window up to the diagonal.
// The grid is persistent: one CTA per SM walks the items (longest first), and for the tensor cores their tiles are one
// sequence: a slot's first S product of an item follows its last P V product of the one before, while the epilogue
// warpgroup still reads the finished O.
//
//   warps 0-3    softmax + correction for slot 0 (thread = query row)
//   warps 4-7    the same for slot 1
//   warps 8-11   epilogue: O / l through shared memory to global, in whole 128-byte lines; LSE
//   warp 12      TMA producer (per item Q of both slots; V_j and K_{j+1} as a pair, two pairs in flight)
//   warp 13      MMA issuer (one elected thread);  warps 14-15 only give their registers away
//
// TMEM: S0 @0, S1 @128 (fp32 scores; P, packed bf16, overwrites S in place and is
// the A operand of the second product), O0 @256, O1 @256+HD.
//
// What bounds it: products of 64 cycles each, 2048 cycles a tile of both slots, against about 3100 from one tile to the next: a slot's chain
// (S product, scores from TMEM, maximum, exponentials, P to TMEM, P V product) is longer than the other slot's work covers, and each
// wait of the issuer returns only when its queue of some six products has nearly run dry.  Under sustained load the card's power
// limit comes first: 1.45 GHz at 990 W (the products alone, waiting for nothing, take 1640 us of the 1960 of 16384 causal tokens there).
// An epilogue of its own instead of one in the softmax warps, S of the next item ahead of it, and pairs of tiles
// (one wait and one commit a tile instead of two of each): 32768 summary-attention tokens (32 heads) 776 -> 728 us, 8192 (16 heads)
// 98.3 -> 96.1, causal 8192 (16 heads) 265 -> 263, 16384 (32 heads) 1980 -> 1967; a single item per SM (2 x 700 tokens, 16 heads) 16.4 -> 16.8.
// Slower, all with the same or nearly the same bits: two threads a row (1960 -> 2050), an issuer per slot (2110), exponentials
// taken with the previous maximum while the tile's own is being found (2550), a warp that waits for the operands in the issuer's place (equal on
// causal, 735 on summary attention).
//
// Bar: FlashAttentionForwardSm100 + block-sparse lists in the reference wheel
// (flash_attn/cute/flash_fwd_sm100.py:68 in the flash_attn_cute wheel, summary_attn/interface.py:77-82 in the
// summary_attn wheel).
#include "attn_common.cuh"
#include "host.h"
#include <string.h>

namespace ksa {

constexpr int kFwdThreads = 512;
constexpr int kOutPitch = 144;                // bytes of a staged row of 64 output columns
// Registers a thread after setmaxnreg: 184 * 256 + 64 * 128 + 80 * 128 = 128 * 512, what the block is launched with.  (A score row of
// 128 columns fits 184 without spilling; with 192 + 64 + 64 the issuer spilled, and a reload costs more there than anywhere else.)
constexpr int kSoftmaxRegs = 184, kEpilogueRegs = 64, kIssueRegs = 80;
template <int HD>
struct FwdSmem {
  static constexpr int kTile = 128 * HD * 2;  // bytes of one 128-row tile
  static constexpr int kQ = 2 * kTile;
  static constexpr int kRing = 4 * kTile;     // two pairs: V of a tile, K of the next
  static constexpr int kStat = 2 * 2 * 128 * 8;          // (max, sum) of every row: two slots, two items
  static constexpr int kOut = 128 * kOutPitch;
  static constexpr int kBar = 256;
  static constexpr int kTotal = kQ + kRing + kStat + kOut + kBar + 1024;
};

struct FwdParams {
  AttnShape s;
  float scale_log2;
  bf16* o;  // [B, Lq, Hq, HD]
  long long o_row_stride, o_batch_stride;
  float* lse;  // [B, Hq, Lq], natural log
  int nslot;   // query heads per CTA (2 when Hq/Hkv is even, else 1)
  int* status;
};

// Load a [128 x HD] tile (row = token) of head `h`, batch `b` starting at token `row0`.
template <int HD>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, int row0, int h, int b, uint64_t* bar) {
#pragma unroll
  for (int half = 0; half < HD / 64; ++half) tma_load_4d(dst + half * 16384, m, half * 64, row0, h, b, bar);
}

template <int HD, bool kCp>
__device__ __forceinline__ void attn_fwd_body(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                                              const CUtensorMap& tmKs, const CUtensorMap& tmVs, const FwdParams& p,
                                              const CpSources* cps) {
  using S = FwdSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + S::kQ;
  float2* sStat = reinterpret_cast<float2*>(sKV + S::kRing);       // [slot][item & 1][row]
  uint8_t* sOut = sKV + S::kRing + S::kStat;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + S::kOut);
  uint64_t* q_full = bars;                 // 2: Q of the slot's current work item has landed
  uint64_t* q_empty = q_full + 2;          // 2: every S product of the item has read it
  uint64_t* kv_full = q_empty + 2;          // 2: V of a tile and K of the next one have landed
  uint64_t* kv_empty = kv_full + 2;         // 2: all products of the pair have read it
  uint64_t* s_full = kv_empty + 2;          // 2
  uint64_t* p_full = s_full + 2;            // 4: slot t, first and last keys of the tile
  uint64_t* o_full = p_full + 4;            // 2: the item's last product has been added to O
  uint64_t* o_free = o_full + 2;            // 2: the epilogue has read O
  uint64_t* l_full = o_free + 2;            // 4: slot t, item & 1: the item's row maxima and sums are in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(l_full + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitGuard guard{abort_flag, p.status};
  const AttnShape& sh = p.s;

  // Work items: (query tile, head group, batch), late (long) query tiles first; CTA c takes items c, c + grid, ...
  const int n_qtiles = (sh.Lq + 127) / 128;
  const int heads_per_cta = p.nslot;
  const int n_groups = sh.Hq / heads_per_cta;
  const int per_q = n_groups * sh.B;
  const int n_items = n_qtiles * per_q;
  // round k hands CTA c item k * grid + c, odd rounds in reverse CTA order, which evens out the causal lengths
  auto item_of_round = [&](int k) {
    const int base = k * (int)gridDim.x;
    return base + ((k & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };
  const int n_rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  auto decode = [&](int item, int& q_tile, int& head0, int& b) {
    const int qi = item / per_q, r = item - qi * per_q;
    q_tile = n_qtiles - 1 - qi;
    b = r / n_groups;
    head0 = (r - b * n_groups) * heads_per_cta;
  };
  // key tiles of the next item at or after round k that has any; 0 when there is none left
  auto next_item = [&](int& k) {
    for (; k < n_rounds; ++k) {
      const int item = item_of_round(k);
      if (item >= n_items) continue;
      int q_tile, head0, b;
      decode(item, q_tile, head0, b);
      const int total = key_tiles_for_query_tile(sh, q_tile, b).total();
      if (total > 0) return total;
    }
    return 0;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&kv_full[i], 2); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[2 * i], 128);
      mbar_init(&p_full[2 * i + 1], 128);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_free[i], 4);
      mbar_init(&l_full[2 * i], 4);
      mbar_init(&l_full[2 * i + 1], 4);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 12) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!kCp) grid_dependency_enter();     // the context-parallel form waits for other GPUs: see grid_dependency_enter

  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    if (warp == 12) {
      // -------------------------------------------------------------- TMA producer
      if (elect_one()) {
        // Tiles travel in pairs, V of one with K of the next (of all items in one sequence); the first pair has only K.
        int it = 0;
        uint32_t pair = 0;
        bool ok = true;
        uint32_t waited = 0;   // context parallel: sources whose flag has been seen (bit s: text, bit 2 + s: summary)
        for (int k = 0; k < n_rounds && ok; ++k) {
          const int item = item_of_round(k);
          if (item >= n_items) continue;
          int q_tile, head0, b;
          decode(item, q_tile, head0, b);
          const int kv_head = head0 / (sh.Hq / sh.Hkv);
          const TileRange tr = key_tiles_for_query_tile(sh, q_tile, b);
          const int total = tr.total();
          if (total == 0) continue;
          for (int j = 0; j < total && ok; ++j) {
            const bool is_sum = j < tr.n_sum_tiles;
            const int kt = is_sum ? j : tr.text_first + (j - tr.n_sum_tiles);
            const CUtensorMap* mk = is_sum ? &tmKs : &tmK;
            const CUtensorMap* mv = is_sum ? &tmVs : &tmV;
            int row = kt * 128;
            if (kCp) {
              const int src = is_sum ? (kt * 128) / cps->nsl : (kt * 128 < cps->halo ? 0 : 1);
              row = is_sum ? (kt * 128) % cps->nsl : (src == 0 ? kt * 128 : kt * 128 - cps->halo);
              mk = is_sum ? &cps->ks[src] : &cps->kt[src];
              mv = is_sum ? &cps->vs[src] : &cps->vt[src];
              const uint32_t bit = 1u << (is_sum ? 2 + src : src);
              const uint32_t* flag = is_sum ? cps->sum_flag[src] : cps->text_flag[src];
              if (flag != nullptr && !(waited & bit)) {
                if (!flag_wait_ge(flag, cps->flag_target, p.status, kTimeoutPeerFlag, true)) {
                  *abort_flag = 1;
                  ok = false;
                  break;
                }
                waited |= bit;
              }
            }
            if (pair == 0) {
              mbar_arrive(&kv_full[0]);
            }
            mbar_expect_tx(&kv_full[pair & 1], S::kTile);
            load_tile<HD>(sKV + ((pair & 1) * 2 + 1) * S::kTile, mk, row, kv_head, b, &kv_full[pair & 1]);
            // a slot's Q is replaced once the previous item's last S product has read it
            if (j == 0) {
              for (int t = 0; t < heads_per_cta && ok; ++t) {
                if (!mbar_wait(&q_empty[t], (it & 1) ^ 1, guard, kTimeoutStageEmpty)) { ok = false; break; }
                mbar_expect_tx(&q_full[t], S::kTile);
                load_tile<HD>(sQ + t * S::kTile, &tmQ, q_tile * 128, head0 + t, b, &q_full[t]);
              }
              if (!ok) break;
            }
            ++pair;
            if (!mbar_wait(&kv_empty[pair & 1], ((pair >> 1) & 1) ^ 1, guard, kTimeoutStageEmpty)) { ok = false; break; }
            mbar_expect_tx(&kv_full[pair & 1], S::kTile);
            load_tile<HD>(sKV + (pair & 1) * 2 * S::kTile, mv, row, kv_head, b, &kv_full[pair & 1]);
          }
          ++it;
        }
        if (ok && it > 0) mbar_arrive(&kv_full[pair & 1]);      // the last pair has no K
      }
    } else if (warp == 13) {
      // -------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
        constexpr uint32_t idesc_o = umma_idesc_bf16(128, HD, 0, 1);
        const uint64_t q_desc = smem_desc_kmajor_sw128(smem_u32(sQ)), k_desc = smem_desc_kmajor_sw128(smem_u32(sKV) + S::kTile);
        const uint64_t v_desc = smem_desc_mnmajor_sw128(smem_u32(sKV), 16384);
        auto issue_s = [&](int t, uint32_t pair) {
          const uint64_t qd = q_desc + t * (S::kTile >> 4), kd = k_desc + (pair & 1) * (S::kTile >> 3);
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t off = ((kk / 4) * 16384 + (kk % 4) * 32) >> 4;
            umma_ss(tmem_base + t * 128, qd + off, kd + off, idesc_s, kk != 0);
          }
          umma_commit(&s_full[t]);
        };
        // One sequence of key tiles over all items: a slot's S product of tile i + 1 follows its P V product of tile i, whether
        // both belong to one item or not.
        int round = 0, total = next_item(round);
        bool ok = total > 0;
        if (ok) {
          ok = mbar_wait(&kv_full[0], 0, guard, kTimeoutTmaFull);
          for (int t = 0; t < heads_per_cta && ok; ++t) {
            ok = mbar_wait(&q_full[t], 0, guard, kTimeoutTmaFull);
            if (!ok) break;
            tc_fence_after();
            issue_s(t, 0);
            if (total == 1) umma_commit(&q_empty[t]);
          }
          if (ok) umma_commit(&kv_empty[0]);
        }
        bool first = true;
        int j = 0;
        uint32_t it = 0;
        for (uint32_t step = 0; ok; ++step) {
          const uint32_t pair = step + 1;
          const bool last = j + 1 == total;
          if (last) {
            ++round;
            total = next_item(round);
            j = -1;
          }
          if (!mbar_wait(&kv_full[pair & 1], (pair >> 1) & 1, guard, kTimeoutTmaFull)) break;
          for (int t = 0; t < heads_per_cta; ++t) {
            // the next item's S product follows: its Q is there
            if (last && total > 0 && !mbar_wait(&q_full[t], (it + 1) & 1, guard, kTimeoutTmaFull)) { ok = false; break; }
            // the first product of an item overwrites O: the previous item's epilogue must have read it
            if (first && it > 0 && !mbar_wait(&o_free[t], (it - 1) & 1, guard, kTimeoutSoftmax)) { ok = false; break; }
            if (!mbar_wait(&p_full[2 * t], step & 1, guard, kTimeoutSoftmax)) { ok = false; break; }
            tc_fence_after();
            const uint64_t vd = v_desc + (pair & 1) * (S::kTile >> 3);
            const uint32_t tS = tmem_base + t * 128, tO = tmem_base + 256 + t * HD;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) umma_ts(tO, tS + kk * 8, vd + kk * 128, idesc_o, !first || kk != 0);
            if (!mbar_wait(&p_full[2 * t + 1], step & 1, guard, kTimeoutSoftmax)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int kk = 4; kk < 8; ++kk) umma_ts(tO, tS + kk * 8, vd + kk * 128, idesc_o, 1);
            if (last) umma_commit(&o_full[t]);
            if (total > 0) {
              issue_s(t, pair);
              if (j + 2 == total) umma_commit(&q_empty[t]);
            }
          }
          if (!ok || total == 0) break;
          umma_commit(&kv_empty[pair & 1]);
          first = last;
          if (last) ++it;
          ++j;
        }
      }
    }
  } else if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    // ---------------------------------------------------------------- epilogue: O / l -> global, LSE
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    uint8_t* stage = sOut + quad * 32 * kOutPitch;
    int it = 0;
    bool ok = true;
    for (int k = 0; k < n_rounds && ok; ++k) {
      const int item = item_of_round(k);
      if (item >= n_items) continue;
      int q_tile, head0, b;
      decode(item, q_tile, head0, b);
      const int total = key_tiles_for_query_tile(sh, q_tile, b).total();
      if (total > 0) {
        int next = k + 1;
        if (next_item(next) == 0) continue;        // the last one: see below
      }
      const int q0 = q_tile * 128 + quad * 32, rows = min(32, sh.Lq - q0);       // rows of this warp, <= 0 past the end
      for (int t = 0; t < heads_per_cta; ++t) {
        const int head = head0 + t;
        bf16* dst = p.o + (long long)b * p.o_batch_stride + (long long)q0 * p.o_row_stride + (long long)head * HD;
        float m = 0.f, l = 0.f;
        if (total > 0) {
          if (!mbar_wait(&l_full[2 * t + (it & 1)], (it >> 1) & 1, guard, kTimeoutSoftmax)) { ok = false; break; }
          const float2 ml = sStat[(t * 2 + (it & 1)) * 128 + r];
          m = ml.x;
          l = ml.y;
          if (!mbar_wait(&o_full[t], it & 1, guard, kTimeoutAccFull)) { ok = false; break; }
          tc_fence_after();
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const uint32_t tO = tmem_base + ((uint32_t)(quad * 32) << 16) + 256 + t * HD;
#pragma unroll
        for (int h = 0; h < HD / 64; ++h) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t o[16];
            if (total > 0) {
              tmem_ld16(tO + h * 64 + c * 16, o);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = 0;
            }
#pragma unroll
            for (int i = 0; i < 16; i += 8) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
              v.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
              v.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
              v.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
              *reinterpret_cast<uint4*>(stage + lane * kOutPitch + c * 32 + i * 2) = v;
            }
          }
          if (h == HD / 64 - 1) tc_fence_before();
          __syncwarp();
          if (h == HD / 64 - 1 && lane == 0 && total > 0) mbar_arrive(&o_free[t]);
#pragma unroll 2
          for (int i = 0; i < 8; ++i) {
            const int row = i * 4 + (lane >> 3);
            if (row < rows)
              *reinterpret_cast<uint4*>(dst + row * p.o_row_stride + h * 64 + (lane & 7) * 8) =
                  *reinterpret_cast<const uint4*>(stage + row * kOutPitch + (lane & 7) * 16);
          }
          __syncwarp();
        }
        if (lane < rows && p.lse)
          p.lse[((long long)b * sh.Hq + head) * sh.Lq + q0 + lane] =
              (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
      if (total > 0) ++it;
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
    // ---------------------------------------------------------------- softmax and rescaling
    const int t = warp >> 2;  // slot
    if (t < heads_per_cta) {
      const int quad = warp & 3;
      const int r = quad * 32 + lane;               // row inside the tile
      const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
      const uint32_t tS = tmem_base + lane_addr + t * 128;
      const uint32_t tO = tmem_base + lane_addr + 256 + t * HD;
      uint32_t step = 0;
      int it = 0;
      bool ok = true;
      for (int k = 0; k < n_rounds && ok; ++k) {
        const int item = item_of_round(k);
        if (item >= n_items) continue;
        int q_tile, head0, b;
        decode(item, q_tile, head0, b);
        const TileRange tr = key_tiles_for_query_tile(sh, q_tile, b);
        const int total = tr.total();
        if (total == 0) continue;
        const int q_local = q_tile * 128 + r;
        const int t_glob = sh.q_off + q_local;
        float m_run = -INFINITY, l_run = 0.f;
        const int doc_start = (sh.q_doc_start && q_local < sh.Lq) ? sh.q_doc_start[(long long)b * sh.Lq + q_local] : 0;
        for (int j = 0; j < total; ++j, ++step) {
          // what this row may see of the tile does not depend on the scores: worked out before they arrive
          const bool is_sum = j < tr.n_sum_tiles;
          const int kt = is_sum ? j : tr.text_first + (j - tr.n_sum_tiles);
          int lo, hi;
          allowed_columns(sh, t_glob, is_sum, kt, lo, hi, doc_start);
          const bool row_masked = lo > 0 || hi < 127;
          if (!mbar_wait(&s_full[t], step & 1, guard, kTimeoutAccFull)) { ok = false; break; }
          tc_fence_after();
          uint32_t sreg[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, sreg[c]);
          tmem_wait_ld();
          if (row_masked) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int col = c * 32 + i;
                if (col < lo || col > hi) sreg[c][i] = 0xff800000u;  // -inf; its exponential is an exact 0
              }
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 32; i += 2)
#pragma unroll
            for (int c = 0; c < 4; ++c)
              mx[c] = max3(mx[c], __uint_as_float(sreg[c][i]), __uint_as_float(sreg[c][i + 1]));
          const float m_new = fmaxf(m_run, fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]) * p.scale_log2);  // scale > 0
          if (j == 0) {
            m_run = m_new;
          } else {
            // O is complete up to the previous tile: its product was issued before the S product that has just arrived
            const bool need = m_new > m_run + 8.f;
            if (__any_sync(0xffffffffu, need)) {
              const float alpha = need ? fast_exp2(m_run - m_new) : 1.f;
#pragma unroll 1
              for (int c = 0; c < HD / 16; ++c) {
                uint32_t o[16];
                tmem_ld16(tO + c * 16, o);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                tmem_st16(tO + c * 16, o);
              }
              tmem_wait_st();
              l_run *= alpha;
              if (need) m_run = m_new;
            }
          }
          const float m_use = (m_run == -INFINITY) ? 0.f : m_run;
          const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2), nm2 = f2_pack(-m_use, -m_use);
          uint64_t acc0 = f2_pack(0.f, 0.f), acc1 = acc0;
          // P = 2^(S * scale - m) -> bf16 over the first half of the columns of S; the product P V starts on the
          // first keys while the exponentials of the others are still being computed
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float p0, p1;
              f2_unpack(f2_fma(f2_pack(__uint_as_float(sreg[c][2 * i]), __uint_as_float(sreg[c][2 * i + 1])), sc2, nm2),
                        p0, p1);
              p0 = fast_exp2(p0);
              p1 = fast_exp2(p1);
              if (i & 1) acc1 = f2_add(acc1, f2_pack(p0, p1)); else acc0 = f2_add(acc0, f2_pack(p0, p1));
              pk[i] = pack_bf16x2(p0, p1);
            }
            tmem_st16(tS + c * 16, pk);
            if (c & 1) {
              tmem_wait_st();
              tc_fence_before();
              mbar_arrive(&p_full[t * 2 + (c >> 1)]);
            }
          }
          float lsum, l1;
          f2_unpack(f2_add(acc0, acc1), lsum, l1);
          l_run += lsum + l1;
        }
        if (!ok) break;
        int next = k + 1;
        if (next_item(next) > 0) {
          sStat[(t * 2 + (it & 1)) * 128 + r] = make_float2(m_run, l_run);
          __syncwarp();
          if (lane == 0) mbar_arrive(&l_full[2 * t + (it & 1)]);
          ++it;
          continue;
        }
        // The last item: nothing is left to overlap the epilogue with, so both slots' warps write their rows at the same time.
        if (!mbar_wait(&o_full[t], it & 1, guard, kTimeoutAccFull)) break;
        tc_fence_after();
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        const int head = head0 + t;
        bf16* dst = p.o + (long long)b * p.o_batch_stride + (long long)q_local * p.o_row_stride + (long long)head * HD;
        uint32_t o[HD / 32][32];
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) tmem_ld32(tO + c * 32, o[c]);
        tmem_wait_ld();
        if (q_local < sh.Lq) {
#pragma unroll
          for (int c = 0; c < HD / 32; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(o[c][i]) * inv, __uint_as_float(o[c][i + 1]) * inv);
              v.y = pack_bf16x2(__uint_as_float(o[c][i + 2]) * inv, __uint_as_float(o[c][i + 3]) * inv);
              v.z = pack_bf16x2(__uint_as_float(o[c][i + 4]) * inv, __uint_as_float(o[c][i + 5]) * inv);
              v.w = pack_bf16x2(__uint_as_float(o[c][i + 6]) * inv, __uint_as_float(o[c][i + 7]) * inv);
              *reinterpret_cast<uint4*>(dst + c * 32 + i) = v;
            }
          if (p.lse)
            p.lse[((long long)b * sh.Hq + head) * sh.Lq + q_local] =
                (l_run > 0.f) ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmKs,
                const __grid_constant__ CUtensorMap tmVs, FwdParams p) {
  attn_fwd_body<HD, false>(tmQ, tmK, tmV, tmKs, tmVs, p, nullptr);
}

// The same kernel for one shard of a context-parallel group: keys and values come from the sources in `cps`.
template <int HD>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_cp_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CpSources cps, FwdParams p) {
  attn_fwd_body<HD, true>(tmQ, cps.kt[1], cps.vt[1], cps.ks[0], cps.vs[0], p, &cps);
}

// [B, T, H, HD] view -> 4-D tensor map {HD, T, H, B}, box {64, 128, 1, 1}, 128-byte swizzle.
static int make_head_tmap(CUtensorMap* m, const void* base, int HD, long long T, int H, int B, long long row_stride,
                          long long batch_stride) {
  uint64_t dims[4] = {(uint64_t)HD, (uint64_t)(T > 0 ? T : 1), (uint64_t)H, (uint64_t)B};
  uint64_t str[4] = {2, (uint64_t)row_stride * 2, (uint64_t)HD * 2, (uint64_t)batch_stride * 2};
  uint32_t box[4] = {64, 128, 1, 1};
  return make_tmap(m, base, 2, 4, dims, str, box, true);
}

template <int HD>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tks,
                      const CUtensorMap& tvs, const FwdParams& p, cudaStream_t st) {
  auto kern = attn_fwd_kernel<HD>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, FwdSmem<HD>::kTotal));
  const int items = ((p.s.Lq + 127) / 128) * (p.s.Hq / p.nslot) * p.s.B;
  int sms = sm_count();
  if (sms <= 0) return 1;
  dim3 grid(items < sms ? items : sms);
  KSA_CHECK_CUDA(launch_kernel(kern, grid, dim3(kFwdThreads), (size_t)FwdSmem<HD>::kTotal, st, tq, tk, tv, tks, tvs, p));
  return 0;
}

template <int HD>
static int launch_fwd_cp(const CUtensorMap& tq, const CpSources& cps, const FwdParams& p, cudaStream_t st) {
  auto kern = attn_fwd_cp_kernel<HD>;
  static PerDevice raised;
  KSA_CHECK_CUDA(raise_smem_limit(raised, kern, FwdSmem<HD>::kTotal));
  const int items = ((p.s.Lq + 127) / 128) * (p.s.Hq / p.nslot) * p.s.B;
  int sms = sm_count();
  if (sms <= 0) return 1;
  dim3 grid(items < sms ? items : sms);
  kern<<<grid, kFwdThreads, FwdSmem<HD>::kTotal, st>>>(tq, cps, p);
  KSA_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace ksa

// Text-query attention forward of ONE SHARD of a context-parallel group, reading keys and values where they are.
// q, o, lse: this rank's queries and outputs as in ksa_attn_fwd.  Keys / values: `text_src[0]` = first halo row in the
// previous rank's exchange slot (ignored when halo = 0), `text_src[1]` = this rank's own text rows, `sum_src[s]` =
// the summary rows of rank s (s < n_sum_src - 1: peers; the last one: this rank); every source is a [B, rows, 2*Hkv*HD]
// block, K in the first Hkv*HD columns and V in the rest, row stride `src_rs`, batch strides `text_bs` / `sum_bs`
// (elements).  `halo` and `nsl` (summary rows per rank) must be multiples of 128 unless there is no halo / a single
// summary source.  `text_flags[s]` / `sum_flags[s]`: address of a flag in this rank's memory that the owner of the
// source raises to `flag_target` when its slot is filled, or null for sources that need no wait.
// Peer memory is only ever read with TMA loads issued by this kernel's own CTAs (no multicast).
KSA_API int ksa_attn_fwd_cp(const void* q, void* o, void* lse, int B, int Hq, int Hkv, int HD, int Lq, long long q_rs,
                            long long q_bs, long long o_rs, long long o_bs, const void* const* text_src, int halo,
                            int local_rows, const void* const* sum_src, int n_sum_src, int nsl, long long src_rs,
                            long long text_bs, long long sum_bs, const void* const* text_flags,
                            const void* const* sum_flags, unsigned flag_target, int q_off, int k_off, int chunk,
                            int n_sum, int window, int tok_window, float scale, void* stream) {
  KSA_ENTER(q);
  using namespace ksa;
  KSA_REQUIRE(HD == 128 || HD == 64, "attn_fwd_cp: head_dim %d unsupported (64 or 128)", HD);
  KSA_REQUIRE(Hq % Hkv == 0 && chunk > 0, "attn_fwd_cp: bad head counts / chunk");
  KSA_REQUIRE(halo >= 0 && halo % 128 == 0, "attn_fwd_cp: halo %d must be a multiple of 128", halo);
  KSA_REQUIRE(n_sum_src >= 0 && n_sum_src <= kCpMaxSum, "attn_fwd_cp: %d summary sources (max %d)", n_sum_src, kCpMaxSum);
  KSA_REQUIRE(n_sum_src <= 1 || nsl % 128 == 0, "attn_fwd_cp: %d summary rows per rank must be a multiple of 128", nsl);
  KSA_REQUIRE(o_rs % 8 == 0, "attn_fwd_cp: output row stride must be a multiple of 8");
  if (B == 0 || Lq == 0) return 0;
  CUtensorMap tq;
  CpSources cps;
  memset(&cps, 0, sizeof(cps));
  int rc;
  if ((rc = make_head_tmap(&tq, q, HD, Lq, Hq, B, q_rs, q_bs))) return rc;
  const long long voff = (long long)Hkv * HD;
  for (int s = 0; s < 2; ++s) {
    const int rows = s == 0 ? halo : local_rows;
    const bf16* base = static_cast<const bf16*>(text_src[rows > 0 ? s : 1]);
    if ((rc = make_head_tmap(&cps.kt[s], base, HD, rows > 0 ? rows : 1, Hkv, B, src_rs, text_bs))) return rc;
    if ((rc = make_head_tmap(&cps.vt[s], base + voff, HD, rows > 0 ? rows : 1, Hkv, B, src_rs, text_bs))) return rc;
    cps.text_flag[s] = text_flags ? static_cast<const uint32_t*>(text_flags[s]) : nullptr;
  }
  for (int s = 0; s < kCpMaxSum; ++s) {
    const int src = s < n_sum_src ? s : (n_sum_src > 0 ? n_sum_src - 1 : -1);
    const bf16* base = src >= 0 ? static_cast<const bf16*>(sum_src[src]) : static_cast<const bf16*>(text_src[1]);
    if ((rc = make_head_tmap(&cps.ks[s], base, HD, nsl > 0 ? nsl : 1, Hkv, B, src_rs, sum_bs))) return rc;
    if ((rc = make_head_tmap(&cps.vs[s], base + voff, HD, nsl > 0 ? nsl : 1, Hkv, B, src_rs, sum_bs))) return rc;
    cps.sum_flag[s] = (sum_flags && s < n_sum_src) ? static_cast<const uint32_t*>(sum_flags[s]) : nullptr;
  }
  cps.flag_target = flag_target;
  cps.halo = halo;
  cps.nsl = nsl > 0 ? nsl : 128;
  FwdParams p;
  p.s = AttnShape{B, Hq, Hkv, Lq, halo + local_rows, n_sum_src * nsl, q_off, k_off, 0, chunk, n_sum > 0 ? n_sum : 1,
                  window, tok_window, nullptr, nullptr};
  p.scale_log2 = scale * 1.4426950408889634f;
  p.o = (bf16*)o;
  p.o_row_stride = o_rs;
  p.o_batch_stride = o_bs;
  p.lse = (float*)lse;
  p.nslot = ((Hq / Hkv) % 2 == 0) ? 2 : 1;
  p.status = status_word();
  KSA_REQUIRE(p.status != nullptr, "could not allocate the status word");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return HD == 128 ? launch_fwd_cp<128>(tq, cps, p, st) : launch_fwd_cp<64>(tq, cps, p, st);
}

// Text-query attention forward.  All tensors are bf16 with the head dimension contiguous:
//   q  [B, Lq, Hq, HD]   (row stride q_rs elements, batch stride q_bs)
//   k,v  [B, Lk, Hkv, HD]  text keys;   ks,vs [B, Ns, Hkv, HD] summary keys (Ns may be 0)
//   o  [B, Lq, Hq, HD];  lse [B, Hq, Lq] fp32 (natural log) or null
// window >= 2^29 disables the chunk window (plain causal); tok_window > 0 adds a token sliding window.
// q_doc_start / k_doc_end (int32 [B, Lq] / [B, Lk], both or neither): packed documents, see AttnShape.
KSA_API int ksa_attn_fwd(const void* q, const void* k, const void* v, const void* ks, const void* vs, void* o,
                         void* lse, int B, int Hq, int Hkv, int HD, int Lq, int Lk, int Ns, long long q_rs,
                         long long q_bs, long long k_rs, long long k_bs, long long v_rs, long long v_bs,
                         long long ks_rs, long long ks_bs, long long vs_rs, long long vs_bs, long long o_rs,
                         long long o_bs, int q_off, int k_off, int s_off, int chunk, int n_sum, int window,
                         int tok_window, float scale, const void* q_doc_start, const void* k_doc_end, void* stream) {
  KSA_ENTER(q);
  using namespace ksa;
  KSA_REQUIRE(HD == 128 || HD == 64, "attn_fwd: head_dim %d unsupported (64 or 128)", HD);
  KSA_REQUIRE(Hq % Hkv == 0, "attn_fwd: Hq %% Hkv != 0");
  KSA_REQUIRE(chunk > 0 && n_sum >= 0, "attn_fwd: bad chunk/n_sum");
  KSA_REQUIRE(o_rs % 8 == 0, "attn_fwd: output row stride must be a multiple of 8");
  if (B == 0 || Lq == 0) return 0;
  CUtensorMap tq, tk, tv, tks, tvs;
  int rc;
  if ((rc = make_head_tmap(&tq, q, HD, Lq, Hq, B, q_rs, q_bs))) return rc;
  if ((rc = make_head_tmap(&tk, k, HD, Lk, Hkv, B, k_rs, k_bs))) return rc;
  if ((rc = make_head_tmap(&tv, v, HD, Lk, Hkv, B, v_rs, v_bs))) return rc;
  if (Ns > 0) {
    if ((rc = make_head_tmap(&tks, ks, HD, Ns, Hkv, B, ks_rs, ks_bs))) return rc;
    if ((rc = make_head_tmap(&tvs, vs, HD, Ns, Hkv, B, vs_rs, vs_bs))) return rc;
  } else {
    tks = tk;
    tvs = tv;
  }
  FwdParams p;
  p.s = AttnShape{B, Hq, Hkv, Lq, Lk, Ns, q_off, k_off, s_off, chunk, n_sum > 0 ? n_sum : 1, window, tok_window,
                  (const int*)q_doc_start, (const int*)k_doc_end};
  p.scale_log2 = scale * 1.4426950408889634f;
  p.o = (bf16*)o;
  p.o_row_stride = o_rs;
  p.o_batch_stride = o_bs;
  p.lse = (float*)lse;
  p.nslot = ((Hq / Hkv) % 2 == 0) ? 2 : 1;
  p.status = status_word();
  KSA_REQUIRE(p.status != nullptr, "could not allocate the status word");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return HD == 128 ? launch_fwd<128>(tq, tk, tv, tks, tvs, p, st) : launch_fwd<64>(tq, tk, tv, tks, tvs, p, st);
}
