// Attention forward at head_dim 256: one persistent CTA per SM, one query tile of 128 rows at a time, blocks of 128 keys.
//   warps 0-3, 4-7   softmax: warpgroup h takes keys [64 h, 64 h + 64) of every block; thread = row = TMEM lane
//   warp  8          TMA producer of Q, K and V, tile scheduler
//   warp  9          MMA issuer: S = Q K^T (operands in shared memory), O += P V (P read from TMEM)
// TMEM (512 columns): S 128, two buffers of 64 for the 16-bit P, O 256.
//
// What bounds it and why this shape.  Per block of 128 keys the tensor pipe needs 16 x 64 clk for S and 8 x 128 for P V, 2048 in all,
// the special-function unit 1024; a block takes 3100 clk with the soft-cap and 2830 without (a launch of 85.6 blocks per SM, everything
// included; with two S buffers, below, 3130 and 2900): no pipe is full, the chain S -> softmax -> P -> P V of one tile is what is left, and
// in long launches the power limit.
// S is free as soon as the softmax warps have it in registers, so that S(n+1) is computed under the softmax of block n and before
// P V(n).  With two S buffers, in which P took S's place, S(n+2) had to wait for P V(n) (us, before -> now, bf16, no soft-cap): 16/8 heads,
// causal, 1024 tokens 18.23 -> 18.02, 4096 tokens 110.5 -> 106.5, 8192 tokens 405.2 -> 398.7; 500 queries on 4000 keys, 32/8 heads 50.9 ->
// 49.9; 4 x 1500 tokens 80.5 -> 78.9; with the soft-cap, where the softmax is longer, equal.  With 64-key blocks and one softmax
// warpgroup a block cost every hand-over of that chain twice as often, and one warp per SM sub-partition could not keep up with the
// soft-cap.  S with N = 128 runs at the full rate with Q in shared memory (N = 64: 48 instead of 32 clk), so Q needs no TMEM and S
// holds 128 keys.
// Measured, 64-key blocks -> 128-key blocks (one box, bf16, us, idle GPU): 16/8 heads, 8192 tokens, window 4096, soft-cap 50: 376 -> 330; 500 queries
// on 4000 keys, 32/8 heads: 52.4 -> 50.7, with soft-cap 64.9 -> 53.8; 16/8 heads, causal, 8192 tokens 402 -> 391, 1024 tokens 19.1 -> 18.3,
// with soft-cap 23.0 -> 19.7, 64 tokens 6.6 -> 6.7.  In a loop under the power cap: window 4096, soft-cap 447 -> 396.
#pragma once

#include "attn_fwd_persist.cuh"
#include "attn_pair.h"

namespace b200 {

struct SplitCfg {
  static constexpr int D = 256, BM = 128, BN = 128, PB = 2;   // PB: P buffers
  static constexpr int COLS = BN / 2;                // keys of a softmax thread
  static constexpr int KSUB = D / 64;                // 64-element (128-byte) column blocks of a row
  static constexpr int Q_TILE_BYTES = BM * D * 2;
  // One ring of 32 KB stages.  A K block is two stages of 128 keys x 128 dims, a V block two of 64 keys x 256 dims: each stage is a
  // complete operand of a run of eight (four) MMAs.
  static constexpr int STAGE_BYTES = 32768, PARTS = 2, V_KEYS = BN / PARTS, SLOTS = 5;
  static constexpr int P_COL = BN, O_COL = P_COL + PB * BN / 2, TMEM_COLS = 512;
  static_assert(O_COL + D == TMEM_COLS, "TMEM plan");
  static constexpr int SOFTMAX_WARPS = 8, PRODUCER_WARP = 8, THREADS = 320;
  // barriers
  static constexpr int BAR_Q_FULL = 0;
  static constexpr int BAR_Q_FREE = 1;                       // last S of a tile retired
  static constexpr int BAR_S_FULL = 2;
  static constexpr int BAR_S_FREE = 3;                       // S is in the registers of the eight softmax warps
  static constexpr int BAR_P_FULL = 4;                       // [PB] eight softmax warps
  static constexpr int BAR_O_FULL = BAR_P_FULL + PB;         // [2] P V of block g completes barrier g % 2
  static constexpr int BAR_FULL = BAR_O_FULL + 2;            // [SLOTS]
  static constexpr int BAR_EMPTY = BAR_FULL + SLOTS;         // [SLOTS]
  static constexpr int BAR_SCHED = BAR_EMPTY + SLOTS;        // [2] item of slot k % 2 published
  static constexpr int BAR_SCHED_FREE = BAR_SCHED + 2;       // [2] read by the softmax warps and the issuer
  static constexpr int BAR_DRAIN = BAR_SCHED_FREE + 2;
  static constexpr int NUM_BARS = BAR_DRAIN + 1;
  // behind the tiles: barriers, [half][row] floats (maxima and sums handed between a row's two threads), TMEM address, abort flag, two
  // scheduler slots, skip flag
  static constexpr int OFF_BARS = Q_TILE_BYTES + SLOTS * STAGE_BYTES;
  static constexpr int OFF_XCH = OFF_BARS + (NUM_BARS * 8 + 15) / 16 * 16;
  static constexpr int OFF_MISC = OFF_XCH + 2 * BM * 4;
  static constexpr int SMEM_BYTES = OFF_MISC + 32 + 1024;    // +1024: manual alignment
  static_assert(SMEM_BYTES <= 232448, "shared memory budget exceeded");
};

// Blocks of one query tile, whose visible key range [lo, hi) is in half blocks: the first block starts at the first visible half, so
// only the last one can be half a block.  For that one there is no second V stage, no P V of its second half and no work for the second
// warpgroup.  In whole blocks only, short prompts and narrow windows paid for up to twice their keys (us, whole -> with a half block;
// 16/8 heads): 64 tokens 7.28 -> 6.48, 8 x 40 heads of 64 tokens 15.8 -> 13.0, 8192 tokens with a window of 16 58.8 -> 52.2, of 16 with
// soft-cap 68.6 -> 61.4; calls without a half block keep their times within 2 % (8 x 40 heads, 200 tokens, soft-cap 36.2 -> 36.4).
struct SplitBlocks {
  int count;
  bool half_last;
  __device__ __forceinline__ explicit SplitBlocks(const TileInfo& t) : count((t.hi - t.lo + 1) >> 1), half_last(((t.hi - t.lo) & 1) != 0) {}
};

struct SplitCtx {
  uint8_t* smem;
  uint64_t* bars;
  float* xch;
  volatile int* abort_flag;
  volatile int* sched;   // [2] item index or -1
  volatile int* skip;    // status word of the device at the start
  uint32_t tmem_base;

  __device__ __forceinline__ bool wait(int bar, int parity, int code) const {
    return mbar_wait(&bars[bar], parity & 1, abort_flag, code);
  }
  __device__ __forceinline__ bool wait_warp(int bar, int parity, int code) const {   // one outcome for the whole warp
    return mbar_wait_warp(&bars[bar], parity & 1, abort_flag, code);
  }
};

// The two warps that share a query tile's rows meet in a named barrier (64 threads) that also ORs a predicate.
__device__ __forceinline__ bool pair_vote(int id, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"((uint32_t)pred)
      : "memory");
  return r != 0;
}

// ------------------------------ softmax warps ------------------------------
// Both threads of a row need the same reference maximum m (their P feed one accumulator), but m moves only in a tile's first block
// and where a block's maximum exceeds it by more than 2^8 (lazy rescale).  So the common block costs one vote between the two warps
// of a 32-row group; only after a vote for it are the maxima exchanged through shared memory.
//
// Steps and failure: attn_pair.h.  A warp whose bounded wait ran out takes part in one more step and leaves; its partner leaves in
// that same step.  A warp that is done takes part in one last step.  No named barrier is ever waited for alone.
template <bool BF16, bool SOFTCAP>
struct SplitSoftmax {
  using Cfg = SplitCfg;
  static constexpr int D = Cfg::D, COLS = Cfg::COLS, PB = Cfg::PB;
  const SplitCtx& c;
  const FwdParams& p;
  const int half, warp_q, lane, bar_id;
  const uint32_t lane_addr, o_addr;   // o_addr: this thread's half of the row's O
  float m, l;                         // l: sum of this thread's keys

  __device__ __forceinline__ SplitSoftmax(const SplitCtx& c_, const FwdParams& p_, int warp, int lane_)
      : c(c_), p(p_), half(warp >> 2), warp_q(warp & 3), lane(lane_), bar_id(1 + (warp & 3)),
        lane_addr(c_.tmem_base + ((uint32_t)((warp & 3) * 32) << 16)),
        o_addr(c_.tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + Cfg::O_COL + (warp >> 2) * (D / 2)) {}

  // the operations of attn_pair.h
  __device__ __forceinline__ bool vote(bool x) const { return pair_vote(bar_id, x); }
  __device__ __forceinline__ void put(float x) const { word(half) = x; }
  __device__ __forceinline__ float get() const { return word(half ^ 1); }
  __device__ __forceinline__ volatile float& word(int h) const { return c.xch[h * Cfg::BM + warp_q * 32 + lane]; }

  // The reference maximum moves where a block's maximum asks for it: m, and l and O with it.  False: leave.
  __device__ __forceinline__ bool agree(int n, int g, bool ok, float m_blk) {
    const PairStep step = pair_block(*this, ok, n == 0 || m_blk - m > 8.0f, m_blk);   // exp2(x - m) stays <= 256
    if (step == PairStep::kLeave) return false;
    if (step == PairStep::kMoved) {
      if (n == 0) {
        m = fmaxf(m, m_blk);
      } else {
        float alpha = 1.0f;
        bool rescale = false;
        if (m_blk - m > 8.0f) {
          alpha = ex2_approx(m - m_blk);
          m = m_blk;
          l *= alpha;
          rescale = true;
        }
        if (__any_sync(0xffffffffu, rescale)) {   // the same in both warps: they hold the same rows
          // P V(g-1): its barrier is exactly in or just past the awaited phase -- S(g) complete implies P V(g-2), and P V(g+1) waits
          // for this thread's P(g).
          if (!c.wait_warp(Cfg::BAR_O_FULL + ((g - 1) & 1), (g - 1) >> 1, WAIT_O_FULL)) {
            pair_leave(*this);
            return false;
          }
          tc_fence_after();
          row_rescale<D / 2>(o_addr, alpha);
        }
      }
    }
    return true;
  }
  __device__ __forceinline__ void deliver(int buf) const {
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&c.bars[Cfg::BAR_P_FULL + buf]);
  }

  __device__ __forceinline__ void release_s() const {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&c.bars[Cfg::BAR_S_FREE]);
  }

  // A half block of the second warpgroup: no keys, but its half of O moves with the maximum.
  __device__ __forceinline__ bool block_without_keys(int n, int g) {
    const int buf = g % PB;
    const bool ok = c.wait(Cfg::BAR_S_FULL, g, WAIT_S_FULL);
    tc_fence_after();
    release_s();
    if (!agree(n, g, ok, -INFINITY)) return false;
    deliver(buf);
    return true;
  }

  // One block of one row.  `g` counts the CTA's blocks, n those of the tile.  False: leave (no further step).
  template <bool MASK>
  __device__ __forceinline__ bool block(int n, int g, int lo_c, int hi_c, float cmul) {
    const int buf = g % PB;
    const uint32_t s_addr = lane_addr + half * COLS;
    const uint32_t p_addr = lane_addr + Cfg::P_COL + buf * (Cfg::BN / 2) + half * (COLS / 2);
    const bool ok = c.wait(Cfg::BAR_S_FULL, g, WAIT_S_FULL);
    tc_fence_after();
    uint32_t sr[COLS / 32][32];
#pragma unroll
    for (int ch = 0; ch < COLS / 32; ++ch) tmem_ld32(s_addr + ch * 32, sr[ch]);
    tmem_ld_wait();
    release_s();

    bool cap_poly_only = false;
    const float m_blk = row_maximum<SOFTCAP, MASK, COLS>(sr, lo_c, hi_c, p, cmul, cap_poly_only);
    if (!agree(n, g, ok, m_blk)) return false;
    l += row_exponentials<BF16, SOFTCAP, MASK, COLS>(sr, p_addr, lo_c, hi_c, p, cmul, m, cap_poly_only);
    deliver(buf);
    return true;
  }

  __device__ __forceinline__ void run(const SchedParams& sp) {
    const float cmul = SOFTCAP ? p.cap_out : p.scale_log2;
    int g = 0;
    for (int k = 0;; ++k) {
      if (!c.wait_warp(Cfg::BAR_SCHED + (k & 1), k >> 1, WAIT_SCHED)) {
        pair_leave(*this);
        return;
      }
      const int item = c.sched[k & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(&c.bars[Cfg::BAR_SCHED_FREE + (k & 1)]);   // slot may be rewritten for item k + 2
      if (item < 0) break;
      const TileInfo t = decode_item(item, p, sp, COLS);
      const SplitBlocks blocks(t);
      const int row = t.q0 + warp_q * 32 + lane;
      m = -1.0e30f;   // finite, so that fully masked blocks stay NaN-free
      l = 0.f;
      // visible keys of this row: [lo_key, hi_key]; a block needs element masks only if some row of the tile sees it partially
      const int hi_key = (p.causal ? min(row + p.delta, p.kv_len - 1) : p.kv_len - 1) - half * COLS;
      const int lo_key = ((p.causal && p.window > 0) ? (row + p.delta - p.window + 1) : -(1 << 28)) - half * COLS;
      const int hi_first = p.causal ? min(t.q0 + p.delta, p.kv_len - 1) : p.kv_len - 1;
      const int lo_last = (p.causal && p.window > 0) ? (t.q0 + 127 + p.delta - p.window + 1) : -(1 << 28);
      const int with_keys = blocks.count - (half == 1 && blocks.half_last ? 1 : 0);
      for (int n = 0; n < with_keys; ++n, ++g) {
        const int k0 = t.lo * COLS + n * Cfg::BN;
        const bool need_mask = (hi_first - k0 < Cfg::BN - 1) || (lo_last - k0 > 0);
        const bool go = need_mask ? block<true>(n, g, lo_key - k0, hi_key - k0, cmul) : block<false>(n, g, 0, 0, cmul);
        if (!go) return;
      }
      if (with_keys < blocks.count) {
        if (!block_without_keys(with_keys, g)) return;
        ++g;
      }
      // Epilogue; the issuer is already computing the next tile's S meanwhile.  The next tile's first P V (which overwrites O) is
      // issued only after this warp has delivered that tile's first P, i.e. after the loads below have completed.
      float l_row = l;
      if (!pair_total(*this, [&] { return c.wait(Cfg::BAR_O_FULL + ((g - 1) & 1), (g - 1) >> 1, WAIT_O_FULL); }, l_row)) return;
      tc_fence_after();
      const bool in_range = row < p.q_len;
      row_store<BF16, D / 2>(o_addr, p.out, (((int64_t)t.b * p.q_len + row) * p.heads + t.h) * (int64_t)D + half * (D / 2), l_row, in_range);
      tc_fence_before();
      if (half == 0 && p.lse != nullptr && in_range)
        p.lse[((int64_t)t.b * p.heads + t.h) * p.lse_stride + row] = m + log2f(l_row);
    }
    pair_finish(*this);
  }
};

// ------------------------------- TMA producer -------------------------------
__device__ __forceinline__ void split_load_q(const SplitCtx& c, const CUtensorMap* tm_q, const TileInfo& t) {
  using Cfg = SplitCfg;
  mbar_expect_tx(&c.bars[Cfg::BAR_Q_FULL], Cfg::Q_TILE_BYTES);
#pragma unroll
  for (int ks = 0; ks < Cfg::KSUB; ++ks)
    tma_load_4d(c.smem + ks * (Cfg::BM * 128), tm_q, &c.bars[Cfg::BAR_Q_FULL], ks * 64, t.h, t.q0, t.b);
}
__device__ __forceinline__ void split_load_k(const SplitCtx& c, const CUtensorMap* tm_k, const TileInfo& t, int slot, int n, int part) {
  using Cfg = SplitCfg;
  uint64_t* full = &c.bars[Cfg::BAR_FULL + slot];
  mbar_expect_tx(full, Cfg::STAGE_BYTES);
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
    tma_load_4d(c.smem + Cfg::Q_TILE_BYTES + slot * Cfg::STAGE_BYTES + ks * (Cfg::BN * 128), tm_k, full, part * 128 + ks * 64, t.hk,
                t.lo * Cfg::V_KEYS + n * Cfg::BN, t.b);
}
// Q and the first K block of the CTA's first tile, before the set-up of the CTA is over.
__device__ __forceinline__ void split_first_loads(const SplitCtx& c, const CUtensorMap* tm_q, const CUtensorMap* tm_k, const TileInfo& t) {
  split_load_q(c, tm_q, t);
#pragma unroll
  for (int part = 0; part < SplitCfg::PARTS; ++part) split_load_k(c, tm_k, t, part, 0, part);
}

// One thread.  Ring stages in the order the issuer consumes them: K(0), then K(n+1), V(n) for n = 0, 1, ...
template <bool PERSISTENT>
__device__ __forceinline__ void split_producer(const SplitCtx& c, const CUtensorMap* tm_q, const CUtensorMap* tm_k,
                                               const CUtensorMap* tm_v, const FwdParams& p, const SchedParams& sp) {
  using Cfg = SplitCfg;
  constexpr int SL = Cfg::SLOTS;
  uint8_t* ring = c.smem + Cfg::Q_TILE_BYTES;
  int ring_i = Cfg::PARTS, tiles = 1;   // stages and Q tiles issued so far (split_first_loads)
  bool ok = true;
  for (int k = 0; ok; ++k) {
    // the first tile of a CTA is its own index (no round trip to the counter before the first load is issued)
    int item = k == 0 ? (int)blockIdx.x : sp.total_items;
    if (PERSISTENT && k > 0) item = (int)(gridDim.x + atomicAdd(&sp.counter[0], 1u));
    const bool valid = item < sp.total_items;
    // slot k % 2 still holds item k-2 until every reader has read it
    if (k >= 2 && !c.wait(Cfg::BAR_SCHED_FREE + (k & 1), (k >> 1) - 1, WAIT_SCHED)) {
      ok = false;
      break;
    }
    c.sched[k & 1] = valid ? item : -1;
    mbar_arrive(&c.bars[Cfg::BAR_SCHED + (k & 1)]);
    if (!valid) {
      if constexpr (PERSISTENT) {
        // last CTA out resets the counters for the next launch that uses this pair
        __threadfence();
        const unsigned done = atomicAdd(&sp.counter[1], 1u);
        if (done == gridDim.x - 1) {
          sp.counter[0] = 0;
          sp.counter[1] = 0;
          __threadfence();
        }
      }
      break;
    }
    const TileInfo t = decode_item(item, p, sp, Cfg::V_KEYS);
    const SplitBlocks blocks(t);
    const int nb = blocks.count;
    if (k > 0) {
      ok = c.wait(Cfg::BAR_Q_FREE, k - 1, WAIT_Q_FREE);
      if (!ok) break;
      split_load_q(c, tm_q, t);
      ++tiles;
    }
    auto load = [&](bool is_v, int n) {
#pragma unroll
      for (int part = 0; part < Cfg::PARTS; ++part) {
        if (is_v && part > 0 && blocks.half_last && n == nb - 1) return;
        const int slot = ring_i % SL, use = ring_i / SL;
        if (!ok || (use > 0 && !c.wait(Cfg::BAR_EMPTY + slot, use - 1, is_v ? WAIT_V_EMPTY : WAIT_K_EMPTY))) {
          ok = false;
          return;
        }
        uint64_t* full = &c.bars[Cfg::BAR_FULL + slot];
        if (is_v) {
          mbar_expect_tx(full, Cfg::STAGE_BYTES);
#pragma unroll
          for (int ks = 0; ks < Cfg::KSUB; ++ks)
            tma_load_4d(ring + slot * Cfg::STAGE_BYTES + ks * (Cfg::V_KEYS * 128), tm_v, full, ks * 64, t.hk,
                        t.lo * Cfg::V_KEYS + n * Cfg::BN + part * Cfg::V_KEYS, t.b);
        } else {
          split_load_k(c, tm_k, t, slot, n, part);
        }
        ++ring_i;
      }
    };
    if (k > 0) load(false, 0);
    for (int n = 0; n < nb && ok; ++n) {
      if (n + 1 < nb) load(false, n + 1);
      if (ok) load(true, n);
    }
  }
  if (!ok || *c.abort_flag != 0) {
    // Abort path: do not leave the CTA while our own bulk copies may still be landing in shared memory.  Wait (bounded, 20 ms) for
    // the most recent load of every slot and of Q.
    const uint64_t t0 = global_timer_ns();
    for (int slot = 0; slot < SL; ++slot) {
      if (ring_i <= slot) continue;
      const int last = slot + ((ring_i - 1 - slot) / SL) * SL;   // last stage that used `slot`
      while (!mbar_try_wait(&c.bars[Cfg::BAR_FULL + slot], (last / SL) & 1) && global_timer_ns() - t0 < 20000000ull) {
      }
    }
    while (tiles > 0 && !mbar_try_wait(&c.bars[Cfg::BAR_Q_FULL], (tiles - 1) & 1) && global_timer_ns() - t0 < 20000000ull) {
    }
  }
}

// -------------------------------- MMA issuer --------------------------------
// One warp, an elected lane issues (umma_ss_if):
//   [S(n+1) = Q K(n+1)^T] [O += P V(n)] [S(n+2)] ...
// S(n+1) needs only S(n) in the softmax warps' registers, so it is there when they are done with block n.  P V(n) stays before S(n+2):
// a softmax warp that sees S(n+2) may overwrite P(n).
// The control flow is convergent unless a wait runs out: then one lane may have seen the abort flag and another the barrier's phase.
// Inside of a tile nothing waits for the whole warp, and `ok` is voted on at the end of each tile, so all lanes leave together.
template <bool BF16>
__device__ __forceinline__ void split_issuer(const SplitCtx& c, const FwdParams& p, const SchedParams& sp, int lane) {
  using Cfg = SplitCfg;
  constexpr int SL = Cfg::SLOTS, D = Cfg::D, BN = Cfg::BN, BM = Cfg::BM, PB = Cfg::PB, PARTS = Cfg::PARTS;
  constexpr uint32_t IDESC_PV = make_idesc(BF16, BM, D, false, true);
  // descriptor halves: the upper word is constant, the lower word is (address >> 4) plus a compile-time step
  const uint32_t desc_hi = smem_desc_hi(1024);
  const uint32_t ring = smem_u32(c.smem) + Cfg::Q_TILE_BYTES;
  const uint32_t q_lo = smem_desc_lo(smem_u32(c.smem), 16);
  const uint32_t k_lo = smem_desc_lo(ring, 16);
  const uint32_t v_lo = smem_desc_lo(ring, Cfg::V_KEYS * 128);   // MN-major: LBO = bytes between 64-wide column blocks
  const uint32_t o_tmem = c.tmem_base + Cfg::O_COL;
  const uint32_t elected = elect_one(), bars = smem_u32(c.bars);
  int ring_i = 0, g0 = 0;
  bool ok = true;
  auto wait_full = [&](int i, int code) { return c.wait(Cfg::BAR_FULL + i % SL, i / SL, code); };
  using Whole = std::integral_constant<int, PARTS>;
  using Half = std::integral_constant<int, 1>;
  auto issue_s = [&](auto parts_tag, int gb, bool last_of_tile) {
    constexpr uint32_t IDESC_S = make_idesc(BF16, BM, Cfg::V_KEYS * decltype(parts_tag)::value, false, false);
    const uint32_t s_tmem = c.tmem_base;
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
      const int slot = ring_i % SL;
      if (ok) ok = wait_full(ring_i, WAIT_K_FULL);
      if (part == 0 && ok && gb > 0) ok = c.wait(Cfg::BAR_S_FREE, gb - 1, WAIT_S_FREE);
      ++ring_i;
      if (!ok) return;
      tc_fence_after();
      const uint32_t b0 = k_lo + (uint32_t)(slot * (Cfg::STAGE_BYTES >> 4));
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const int ka = part * 8 + kk;
        const uint32_t a_off = (uint32_t)(((ka / 4) * (BM * 128) + (ka % 4) * 32) >> 4);
        const uint32_t b_off = (uint32_t)(((kk / 4) * (BN * 128) + (kk % 4) * 32) >> 4);
        umma_ss_if<IDESC_S>(elected, s_tmem, q_lo + a_off, b0 + b_off, desc_hi, ka == 0 ? 0u : 1u);
      }
      if (part == PARTS - 1) umma_commit_if(elected, bars + 8 * Cfg::BAR_S_FULL);
      umma_commit_if(elected, bars + 8 * (Cfg::BAR_EMPTY + slot));
      if (part == PARTS - 1 && last_of_tile) umma_commit_if(elected, bars + 8 * Cfg::BAR_Q_FREE);   // no later MMA reads this Q
    }
  };
  auto issue_pv = [&](auto parts_tag, int gb, bool first_of_tile) {
    constexpr int parts = decltype(parts_tag)::value;
    const uint32_t p_tmem = c.tmem_base + Cfg::P_COL + (gb % PB) * (BN / 2);
#pragma unroll
    for (int part = 0; part < parts; ++part) {   // part = half: keys [64 part, 64 part + 64), P in columns [32 part, 32 part + 32)
      const int slot = (ring_i + part) % SL;
      const uint32_t b0 = v_lo + (uint32_t)(slot * (Cfg::STAGE_BYTES >> 4));
#pragma unroll
      for (int kk = 0; kk < Cfg::V_KEYS / 16; ++kk) {
        const uint32_t a = p_tmem + part * (Cfg::COLS / 2) + kk * 8, b = b0 + (uint32_t)(kk * (2048 >> 4));
        umma_ts_if<IDESC_PV>(elected, o_tmem, a, b, desc_hi, (part == 0 && kk == 0 && first_of_tile) ? 0u : 1u);
      }
      umma_commit_if(elected, bars + 8 * (Cfg::BAR_EMPTY + slot));
    }
    // two O barriers in turn: the softmax can run two blocks ahead of the P V products, and a parity wait is exact only while at most
    // one phase of a barrier is outstanding
    umma_commit_if(elected, bars + 8 * (Cfg::BAR_O_FULL + (gb & 1)));
  };
  // P V of one block.  V first: it landed long ago, and nothing but the wait for P should stand before the products.
  auto step_pv = [&](auto parts_tag, int gb, bool first_of_tile) {
    constexpr int parts = decltype(parts_tag)::value;
#pragma unroll
    for (int part = 0; part < parts; ++part)
      if (ok) ok = wait_full(ring_i + part, WAIT_V_FULL);
    if (ok) ok = c.wait(Cfg::BAR_P_FULL + gb % PB, gb / PB, WAIT_P_FULL);
    if (!ok) return;
    tc_fence_after();
    issue_pv(parts_tag, gb, first_of_tile);
    ring_i += parts;
  };
  for (int k = 0; ok; ++k) {
    if (!c.wait_warp(Cfg::BAR_SCHED + (k & 1), k >> 1, WAIT_SCHED)) break;
    const int item = c.sched[k & 1];
    __syncwarp();
    if (lane == 0) mbar_arrive(&c.bars[Cfg::BAR_SCHED_FREE + (k & 1)]);
    if (item < 0) break;
    const TileInfo t = decode_item(item, p, sp, Cfg::V_KEYS);
    const SplitBlocks blocks(t);
    const int nb = blocks.count, whole = nb - (blocks.half_last ? 1 : 0);
    ok = c.wait(Cfg::BAR_Q_FULL, k, WAIT_Q_FULL);
    if (whole > 0 && ok) issue_s(Whole{}, g0, nb == 1);
    for (int n = 0; n + 1 < whole && ok; ++n) {
      issue_s(Whole{}, g0 + n + 1, n + 2 == nb);
      if (ok) step_pv(Whole{}, g0 + n, n == 0);
    }
    // The last whole block and the half block are not in the loop, so that it has no more to decide.
    if (whole < nb && ok) issue_s(Half{}, g0 + whole, true);
    if (whole > 0 && ok) step_pv(Whole{}, g0 + whole - 1, whole == 1);
    if (whole < nb && ok) step_pv(Half{}, g0 + whole, whole == 0);
    ok = __all_sync(0xffffffffu, ok);
    g0 += nb;
  }
  // every MMA issued above has retired before the CTA tears TMEM down
  umma_commit_if(elected, bars + 8 * Cfg::BAR_DRAIN);
  c.wait(Cfg::BAR_DRAIN, 0, WAIT_DRAIN);
}

// PERSISTENT: tiles from the counter; otherwise one tile per CTA (A/B timing).
template <bool BF16, bool SOFTCAP, bool PERSISTENT>
__global__ void __launch_bounds__(SplitCfg::THREADS, 1)
attn_fwd_split_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const FwdParams p, const SchedParams sp) {
  using Cfg = SplitCfg;
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 32) prefetch_l2(&g_device_status);   // read after the wait below
  SplitCtx c;
  c.smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  c.bars = reinterpret_cast<uint64_t*>(c.smem + Cfg::OFF_BARS);
  c.xch = reinterpret_cast<float*>(c.smem + Cfg::OFF_XCH);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(c.smem + Cfg::OFF_MISC);
  c.abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  c.sched = reinterpret_cast<volatile int*>(tmem_slot + 2);
  c.skip = reinterpret_cast<volatile int*>(tmem_slot + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // The producer initialises the barriers, so that its first loads need not wait for the rest of the block.
  const bool producer = warp == Cfg::PRODUCER_WARP && lane == 0;
  if (producer) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
#pragma unroll
    for (int i = 0; i < Cfg::NUM_BARS; ++i) {
      const bool p_full = i >= Cfg::BAR_P_FULL && i < Cfg::BAR_P_FULL + Cfg::PB;
      const bool sched_free = i >= Cfg::BAR_SCHED_FREE && i < Cfg::BAR_SCHED_FREE + 2;
      mbar_init(&c.bars[i], p_full || i == Cfg::BAR_S_FREE ? (uint32_t)Cfg::SOFTMAX_WARPS : sched_free ? (uint32_t)Cfg::SOFTMAX_WARPS + 1u : 1u);
    }
    *c.abort_flag = 0;
    fence_mbar_init();
  }
  TileInfo first_tile;
  if (producer) first_tile = decode_item(blockIdx.x, p, sp, Cfg::V_KEYS);   // the grid has no more CTAs than items
  // The wait comes before the TMEM allocation and the status word: a predecessor that let this launch start early may still have
  // to allocate columns of its own, and what it wrote is visible only now.
  pdl_wait();
  if (producer) {
    fence_proxy_async_global();
    split_first_loads(c, &tm_q, &tm_k, first_tile);
  }
  if (threadIdx.x == 32) *c.skip = *reinterpret_cast<volatile int*>(&g_device_status);
  if (warp == 0) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem_base = *tmem_slot;
  // A launch that follows an expired wait on this device drains immediately (the status word stays set until the host reads it; the
  // tile counter is untouched: the host zeroes it when it clears the word).
  if (*c.skip == 0) {
    if (warp < Cfg::SOFTMAX_WARPS) {
      SplitSoftmax<BF16, SOFTCAP> s(c, p, warp, lane);
      s.run(sp);
    } else if (warp == Cfg::PRODUCER_WARP) {
      if (lane == 0) split_producer<PERSISTENT>(c, &tm_q, &tm_k, &tm_v, p, sp);
    } else {
      split_issuer<BF16>(c, p, sp, lane);
    }
  } else if (producer) {   // the loads above land before the CTA exits (bounded, 20 ms)
    const uint64_t t0 = global_timer_ns();
    for (int bar : {Cfg::BAR_Q_FULL, Cfg::BAR_FULL, Cfg::BAR_FULL + 1})
      while (!mbar_try_wait(&c.bars[bar], 0) && global_timer_ns() - t0 < 20000000ull) {
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(c.tmem_base, Cfg::TMEM_COLS);
}

template <bool BF16, bool SOFTCAP, bool PERSISTENT>
int launch_attn_fwd_split_as(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p,
                             cudaStream_t stream) {
  auto kern = attn_fwd_split_kernel<BF16, SOFTCAP, PERSISTENT>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  B200_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitCfg::SMEM_BYTES));
    configured_dev = dev;
  }
  SchedParams sp;
  const int rc = sched_params(&sp, p, SplitCfg::D, PERSISTENT);
  if (rc != B200_OK) return rc;
  const int grid = PERSISTENT ? std::min(sp.total_items, sm_count()) : sp.total_items;
  B200_CUDA_TRY(launch_kernel(kern, grid, SplitCfg::THREADS, SplitCfg::SMEM_BYTES, stream, 1, tq, tk, tv, p, sp));
  return B200_OK;
}

template <bool BF16, bool SOFTCAP>
int launch_attn_fwd_split(const void* q, const void* k, const void* v, const FwdParams& p, const AttnStrides& st,
                          bool one_tile_per_cta, cudaStream_t stream) {
  using Cfg = SplitCfg;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tensor_map(&tq, q, p.batch, p.q_len, p.heads, Cfg::D, Cfg::BM, BF16, st.q_token, st.q_batch)) != B200_OK ||
      (rc = make_bshd_tensor_map(&tk, k, p.batch, p.kv_len, p.kv_heads, Cfg::D, Cfg::BN, BF16, st.k_token, st.k_batch)) != B200_OK ||
      (rc = make_bshd_tensor_map(&tv, v, p.batch, p.kv_len, p.kv_heads, Cfg::D, Cfg::V_KEYS, BF16, st.v_token, st.v_batch)) !=
          B200_OK)
    return rc;
  return one_tile_per_cta ? launch_attn_fwd_split_as<BF16, SOFTCAP, false>(tq, tk, tv, p, stream)
                          : launch_attn_fwd_split_as<BF16, SOFTCAP, true>(tq, tk, tv, p, stream);
}

}  // namespace b200
