// Fused attention forward for sm_100a:  out = softmax(mask(softcap(q k^T * scale))) v, at head_dim 128 (256: attn_fwd_split.cuh).
//
// One CTA owns NQ query tiles of 128 rows of one (batch, head) and walks the key/value blocks that the
// causal / sliding-window mask leaves visible.  Roles (warp-specialised):
//   warps [0, 4*NQ)      softmax warpgroups, one per query tile: thread r of a group owns row r (TMEM lane r)
//                        -- online softmax, O rescale, epilogue
//   warp  4*NQ           TMA producer: Q once, then K(j), V(j), K(j+1), ... through ONE ring of SLOTS stages
//   warps 4*NQ+1 (+2)    MMA issuers, one per query tile: S = Q K^T (operands in shared memory) and
//                        O += P V (P read from TMEM, V from shared memory) on tcgen05
// TMEM columns: [S tile per query tile (fp32, BN columns; the 16-bit P overwrites its first BN/2 columns)]
//               [O accumulator per query tile (fp32, D columns)].
//
// Reference semantics: deepgengraph_exp/cases/kernels/attn.py:18-34 (mask, scale, fp32 softmax, P rounded to
// the input type before P V) and kernels/gemma2.py:30-34 (soft-cap after the scale, before the mask).
#pragma once

#include "common.cuh"

namespace b200 {

struct FwdParams {
  void* out;    // [B, Sq, H, D]
  float* lse;   // [B*H][lse_stride] base-2 log-sum-exp of the scaled logits, may be null
  int lse_stride;
  int batch, q_len, kv_len, heads, kv_heads;
  int causal, window;
  int delta;          // kv_len - q_len
  float scale_log2;   // scale * log2(e)              (no soft-cap)
  float cap_in;       // scale / softcap              (soft-cap: x = tanh(s * cap_in) * cap_out)
  float cap_out;      // softcap * log2(e)
};

// SB = S buffers per query tile in TMEM.  With SB = 2 the S tile of block j+1 is computed while the softmax of
// block j runs, so a tile's softmax never waits for the tensor pipe in steady state.
template <int BN_, int NQ_, int SB_>
struct FwdCfg {
  static constexpr int D = 128, BN = BN_, NQ = NQ_, SB = SB_;
  static constexpr int BM = 128;
  static constexpr int KSUB = D / 64;                 // 64-element (128-byte) column blocks of a row
  static constexpr int Q_TILE_BYTES = BM * D * 2;
  static constexpr int KV_STAGE_BYTES = BN * D * 2;
  // one ring for K and V blocks (K(j) is item 2n, V(j) item 2n+1): as many slots as fit beside Q, at most 8
  // With one query tile per CTA: TMEM (256 of 512 columns) and shared memory are sized so that TWO
  // CTAs share an SM.  The two are independent (own producer, own issuer, own K/V ring), so one CTA's prologue,
  // epilogue and softmax phases overlap the other's MMAs without any coupling between them.
  static constexpr int CTAS_PER_SM = NQ == 1 ? 2 : 1;
  static constexpr int SMEM_BUDGET = 232448 / CTAS_PER_SM - (CTAS_PER_SM > 1 ? 1024 : 0);   // 1 KB/CTA is reserved by the driver
  static constexpr int SLOTS_FIT = (SMEM_BUDGET - 2048 - NQ * Q_TILE_BYTES) / KV_STAGE_BYTES;
  static constexpr int SLOTS = SLOTS_FIT > 8 ? 8 : SLOTS_FIT;
  static_assert(SLOTS >= 3, "ring too shallow");
  static constexpr int O_BASE = ((NQ * SB * BN + D - 1) / D) * D;
  static constexpr int TMEM_USED = O_BASE + NQ * D;
  static constexpr int TMEM_COLS = TMEM_USED <= 32 ? 32 : TMEM_USED <= 64 ? 64 : TMEM_USED <= 128 ? 128
                                   : TMEM_USED <= 256 ? 256 : 512;
  static_assert(TMEM_USED <= 512, "TMEM budget exceeded");
  // NQ = 2 pads the producer/MMA warps to a full warpgroup so that registers can be re-balanced per warpgroup
  static constexpr int THREADS = NQ == 2 ? 384 : (NQ * 4 + 2) * 32;
  static constexpr bool REBALANCE_REGS = NQ == 2;
  // barrier slots
  static constexpr int BAR_Q_FULL = 0;                       // [NQ]
  static constexpr int BAR_S_FULL = BAR_Q_FULL + NQ;         // [NQ][SB]
  static constexpr int BAR_P_FULL = BAR_S_FULL + NQ * SB;    // [NQ][SB]
  static constexpr int BAR_O_FULL = BAR_P_FULL + NQ * SB;    // [NQ][2]: P V(n) completes O barrier n % 2
  static constexpr int BAR_FULL = BAR_O_FULL + NQ * 2;       // [SLOTS]
  static constexpr int BAR_EMPTY = BAR_FULL + SLOTS;         // [SLOTS]
  static constexpr int BAR_DRAIN = BAR_EMPTY + SLOTS;        // [NQ] one drain barrier per MMA issuer
  static constexpr int BAR_TURN = BAR_DRAIN + NQ;            // [NQ][4]: exp-phase turn of softmax warp w of tile t
  static constexpr int NUM_BARS = BAR_TURN + NQ * 4;
  static constexpr int SMEM_TILES = NQ * Q_TILE_BYTES + SLOTS * KV_STAGE_BYTES;
  static constexpr int SMEM_BYTES = SMEM_TILES + NUM_BARS * 8 + 16 + 1024;  // +1024: manual alignment slack
  static_assert(SMEM_BYTES <= SMEM_BUDGET, "shared memory budget exceeded");
};

// Block range of one query tile: key blocks [lo, hi) hold at least one visible key.
struct TileRange {
  int lo, hi;
};
__device__ __forceinline__ TileRange tile_range(int r_first, int bn, const FwdParams& p) {
  TileRange r;
  if (r_first >= p.q_len) {
    r.lo = r.hi = 0;
    return r;
  }
  const int r_last = min(r_first + 127, p.q_len - 1);
  const int last_key = p.causal ? min(p.kv_len - 1, r_last + p.delta) : p.kv_len - 1;
  r.hi = last_key / bn + 1;
  r.lo = (p.causal && p.window > 0) ? max(0, r_first + p.delta - p.window + 1) / bn : 0;
  return r;
}

template <class Cfg, bool BF16>
struct FwdCtx {
  uint8_t* sQ;
  uint8_t* sKV;
  uint64_t* bars;
  volatile int* abort_flag;
  uint32_t tmem_base;
  int q0, h, hk, b;
  TileRange rng[Cfg::NQ];
  int jmin, jmax;
};

// ------------------------------- TMA producer -------------------------------
template <class Cfg, bool BF16>
__device__ __forceinline__ void fwd_producer(const FwdCtx<Cfg, BF16>& c, const CUtensorMap* tm_q,
                                             const CUtensorMap* tm_k, const CUtensorMap* tm_v) {
  constexpr int SL = Cfg::SLOTS;
  fence_proxy_async_global();
#pragma unroll
  for (int t = 0; t < Cfg::NQ; ++t) {
    if (c.rng[t].hi > c.rng[t].lo) {
      mbar_expect_tx(&c.bars[Cfg::BAR_Q_FULL + t], Cfg::Q_TILE_BYTES);
#pragma unroll
      for (int ks = 0; ks < Cfg::KSUB; ++ks)
        tma_load_4d(c.sQ + t * Cfg::Q_TILE_BYTES + ks * (Cfg::BM * 128), tm_q, &c.bars[Cfg::BAR_Q_FULL + t],
                    ks * 64, c.h, c.q0 + t * Cfg::BM, c.b);
    }
  }
  // Ring items in the order the MMA issuers consume them: K(0..SB-1), then V(n), K(n+SB) for n = 0, 1, ...
  const int nb = c.jmax - c.jmin;
  int issued = 0;
  bool ok = true;
  auto load = [&](bool is_v, int n) {
    const int i = issued, slot = i % SL, use = i / SL;
    if (use > 0 && !mbar_wait(&c.bars[Cfg::BAR_EMPTY + slot], (use - 1) & 1, c.abort_flag, is_v ? WAIT_V_EMPTY : WAIT_K_EMPTY)) {
      ok = false;
      return;
    }
    uint64_t* full = &c.bars[Cfg::BAR_FULL + slot];
    uint8_t* dst = c.sKV + slot * Cfg::KV_STAGE_BYTES;
    const CUtensorMap* tm = is_v ? tm_v : tm_k;
    mbar_expect_tx(full, Cfg::KV_STAGE_BYTES);
#pragma unroll
    for (int ks = 0; ks < Cfg::KSUB; ++ks)
      tma_load_4d(dst + ks * (Cfg::BN * 128), tm, full, ks * 64, c.hk, (c.jmin + n) * Cfg::BN, c.b);
    issued = i + 1;
  };
  for (int n = 0; n < Cfg::SB && n < nb && ok; ++n) load(false, n);
  for (int n = 0; n < nb && ok; ++n) {
    load(true, n);
    if (ok && n + Cfg::SB < nb) load(false, n + Cfg::SB);
  }
  if (!ok || *c.abort_flag != 0) {
    // Abort path: do not leave the CTA while our own bulk copies may still be landing in shared memory.
    // Wait (bounded, 20 ms) for the most recent load of every slot and for the Q tiles.
    const uint64_t t0 = global_timer_ns();
    for (int slot = 0; slot < SL; ++slot) {
      if (issued <= slot) continue;
      const int last = slot + ((issued - 1 - slot) / SL) * SL;   // last item that used `slot`
      const int u = last / SL;
      while (!mbar_try_wait(&c.bars[Cfg::BAR_FULL + slot], u & 1) && global_timer_ns() - t0 < 20000000ull) {
      }
    }
#pragma unroll
    for (int t = 0; t < Cfg::NQ; ++t)
      while (c.rng[t].hi > c.rng[t].lo && !mbar_try_wait(&c.bars[Cfg::BAR_Q_FULL + t], 0) &&
             global_timer_ns() - t0 < 20000000ull) {
      }
  }
}

// -------------------------------- MMA issuer --------------------------------
// One issuing thread PER QUERY TILE (its own warp): the two tiles' chains
//   softmax(j) -> P -> [O += P V(j)] -> [S(j+1) = Q K(j+1)^T] -> softmax(j+1)
// then advance independently, and neither waits behind the other tile's instruction issue.  Both issuers walk
// every key block of the CTA and both arrive on the K/V "stage empty" barriers (count NQ) -- for blocks outside
// a tile's visible range the arrive is immediate.
template <class Cfg, bool BF16, int T>
__device__ __forceinline__ void fwd_mma(const FwdCtx<Cfg, BF16>& c) {
  constexpr int SL = Cfg::SLOTS, D = Cfg::D, BN = Cfg::BN, BM = Cfg::BM, SB = Cfg::SB;
  constexpr uint32_t IDESC_S = make_idesc(BF16, BM, BN, false, false);
  constexpr uint32_t IDESC_PV = make_idesc(BF16, BM, D, false, true);
  // descriptor halves: the upper word is constant, the lower word is (address >> 4) plus a compile-time step
  const uint32_t desc_hi = smem_desc_hi(1024);
  const uint32_t q_lo = smem_desc_lo(smem_u32(c.sQ) + T * Cfg::Q_TILE_BYTES, 16);
  const uint32_t k_lo = smem_desc_lo(smem_u32(c.sKV), 16);
  const uint32_t v_lo = smem_desc_lo(smem_u32(c.sKV), BN * 128);  // MN-major: LBO = bytes between 64-wide column blocks
  const uint32_t s_tmem0 = c.tmem_base + T * SB * BN;             // S buffers; P (packed 16-bit) overwrites the first half
  const uint32_t o_tmem = c.tmem_base + Cfg::O_BASE + T * D;
  const int lo = c.rng[T].lo, hi = c.rng[T].hi;

  auto issue_s = [&](int slot, int buf) {
    const uint32_t b0 = k_lo + (uint32_t)(slot * (Cfg::KV_STAGE_BYTES >> 4));
    const uint32_t s_tmem = s_tmem0 + buf * BN;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      const uint32_t a_off = (uint32_t)(((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4);
      const uint32_t b_off = (uint32_t)(((kk / 4) * (BN * 128) + (kk % 4) * 32) >> 4);
      if (kk == 0)
        umma_ss_c<IDESC_S, 0>(s_tmem, q_lo + a_off, b0 + b_off, desc_hi);
      else
        umma_ss_c<IDESC_S, 1>(s_tmem, q_lo + a_off, b0 + b_off, desc_hi);
    }
    umma_commit(&c.bars[Cfg::BAR_S_FULL + T * SB + buf]);
  };
  auto issue_pv = [&](int slot, int buf, int nt) {
    const bool first = nt == 0;
    const uint32_t b0 = v_lo + (uint32_t)(slot * (Cfg::KV_STAGE_BYTES >> 4));
    const uint32_t s_tmem = s_tmem0 + buf * BN;
    // V block: KSUB column blocks of [BN keys][64 dims]; 16 keys = 2048 bytes further down; P: 8 columns per 16 keys
    if (first)
      umma_ts_c<IDESC_PV, 0>(o_tmem, s_tmem, b0, desc_hi);
    else
      umma_ts_c<IDESC_PV, 1>(o_tmem, s_tmem, b0, desc_hi);
#pragma unroll
    for (int kk = 1; kk < BN / 16; ++kk)
      umma_ts_c<IDESC_PV, 1>(o_tmem, s_tmem + kk * 8, b0 + (uint32_t)(kk * (2048 >> 4)), desc_hi);
    // Two O barriers used alternately: the softmax warps can run two blocks ahead of the P V products, and a
    // parity wait is exact only while at most one phase of a barrier is outstanding.
    umma_commit(&c.bars[Cfg::BAR_O_FULL + T * 2 + (nt & 1)]);
  };

  // All 32 lanes walk the loop (warp-uniform), one elected lane issues.  The issuer walks the ring items in
  // producer order -- K(0..SB-1), then V(n), K(n+SB) -- and every slot is waited for (FULL) before this issuer
  // releases it (EMPTY), also for blocks outside the tile's range: an issuer can therefore never run more than
  // the ring depth ahead of the other one, which keeps the count-NQ EMPTY barriers phase-exact.
  bool ok = true;
  int item = 0;
  bool q_ready = false;
  auto k_item = [&](int n) {   // S(j) = Q K(j)^T into buffer (j - lo) % SB
    const int j = c.jmin + n, slot = item % SL, ph = (item / SL) & 1;
    ++item;
    const bool act = j >= lo && j < hi;
    if (elect_one()) B200_TL((3 * 64 + (n & 63)) * 8 + T * 4 + 2);
    if (act && !q_ready) {
      ok = mbar_wait_warp(&c.bars[Cfg::BAR_Q_FULL + T], 0, c.abort_flag, WAIT_Q_FULL);
      q_ready = true;
    }
    ok = ok && mbar_wait_warp(&c.bars[Cfg::BAR_FULL + slot], ph, c.abort_flag, WAIT_K_FULL);
    if (!ok) return;
    tc_fence_after();
    if (elect_one()) {
      B200_TL((3 * 64 + (n & 63)) * 8 + T * 4 + 3);
      if (act) {
        B200_TL((2 * 64 + (n & 63)) * 8 + T * 4 + 2);
        issue_s(slot, (j - lo) % SB);
        B200_TL((2 * 64 + (n & 63)) * 8 + T * 4 + 3);
      }
      umma_commit(&c.bars[Cfg::BAR_EMPTY + slot]);   // K(j) consumed by this tile
    }
    __syncwarp();
  };
  // Steady state, one step per key block n: [O += P(n) V(n)] and [S(n+SB) = Q K(n+SB)^T] are issued back to
  // back by one elected lane.  The ring slots of both operands were filled long before, so their FULL barriers
  // are observed FIRST; the wait for P(n) -- the only barrier that completes late -- comes last, and nothing
  // but a fence stands between its completion and the twelve MMAs.  (tcgen05 issue is synchronous with the
  // tensor pipe once its queue is full, so every barrier round trip between the two GEMMs used to add to the
  // P(n) -> S(n+SB) latency that the softmax of block n+1 has to cover.)
  auto step = [&](int n, int nb) {
    const int jv = c.jmin + n, vslot = item % SL, vph = (item / SL) & 1;
    ++item;
    const bool has_k = n + SB < nb;
    const int jk = c.jmin + n + SB, kslot = item % SL, kph = (item / SL) & 1;
    if (has_k) ++item;
    const bool act_v = jv >= lo && jv < hi;
    const bool act_k = has_k && jk >= lo && jk < hi;
    const int nt = jv - lo, buf = nt % SB;
    if (elect_one()) B200_TL((3 * 64 + (n & 63)) * 8 + T * 4 + 0);
    ok = mbar_wait_warp(&c.bars[Cfg::BAR_FULL + vslot], vph, c.abort_flag, WAIT_V_FULL);
    if (ok && has_k) ok = mbar_wait_warp(&c.bars[Cfg::BAR_FULL + kslot], kph, c.abort_flag, WAIT_K_FULL);
    if (ok && act_k && !q_ready) {
      ok = mbar_wait_warp(&c.bars[Cfg::BAR_Q_FULL + T], 0, c.abort_flag, WAIT_Q_FULL);
      q_ready = true;
    }
    if (ok && act_v) ok = mbar_wait_warp(&c.bars[Cfg::BAR_P_FULL + T * SB + buf], (nt / SB) & 1, c.abort_flag, WAIT_P_FULL);
    if (!ok) return;
    tc_fence_after();
    if (elect_one()) {
      B200_TL((3 * 64 + (n & 63)) * 8 + T * 4 + 1);
      if (act_v) issue_pv(vslot, buf, nt);
      B200_TL((2 * 64 + (n & 63)) * 8 + T * 4 + 1);
      if (act_k) issue_s(kslot, (jk - lo) % SB);
      B200_TL((2 * 64 + (n & 63)) * 8 + T * 4 + 3);
      umma_commit(&c.bars[Cfg::BAR_EMPTY + vslot]);              // V(n) consumed by this tile
      if (has_k) umma_commit(&c.bars[Cfg::BAR_EMPTY + kslot]);   // K(n+SB) consumed by this tile
    }
    __syncwarp();
  };
  const int nb = c.jmax - c.jmin;
  for (int n = 0; n < SB && n < nb && ok; ++n) k_item(n);
  for (int n = 0; n < nb && ok; ++n) step(n, nb);
  // every MMA issued above has retired before the CTA tears TMEM down
  if (elect_one()) umma_commit(&c.bars[Cfg::BAR_DRAIN + T]);
  __syncwarp();
  mbar_wait_warp(&c.bars[Cfg::BAR_DRAIN + T], 0, c.abort_flag, WAIT_DRAIN);
}

// ------------------------------ softmax warpgroup ----------------------------
// 2^x for two values on the FMA/ALU pipes (no special-function unit): round x to the nearest integer n with the
// 1.5 * 2^23 trick, evaluate a cubic minimax polynomial of 2^f on f = x - n in [-0.5, 0.5] (max relative error
// 7.5e-5, far below the 2^-9 rounding of the 16-bit P), and add n to the exponent field.  x is clamped at -125 so
// that the exponent never wraps.  Used for a fixed fraction of the columns of every unmasked block: the
// exponentials of attention are bound by the special-function unit (16 results per clock per SM), and moving
// part of them to the FMA pipe shortens the softmax phase.
__device__ __forceinline__ float2 exp2_poly2(float2 x) {
  const float kMagic = 12582912.0f;  // 1.5 * 2^23
  x.x = fmaxf(x.x, -125.0f);
  x.y = fmaxf(x.y, -125.0f);
  const float2 r = fadd2(x, make_float2(kMagic, kMagic));              // low mantissa bits = round(x)
  const float2 n = fadd2(r, make_float2(-kMagic, -kMagic));            // round(x) as a float
  const float2 f = fadd2(x, make_float2(-n.x, -n.y));                  // in [-0.5, 0.5]
  float2 pl = ffma2(f, make_float2(0.0551716648f, 0.0551716648f), make_float2(0.2426111251f, 0.2426111251f));
  pl = ffma2(pl, f, make_float2(0.6932609677f, 0.6932609677f));
  pl = ffma2(pl, f, make_float2(0.9999280572f, 0.9999280572f));
  float2 out;
  out.x = __uint_as_float(__float_as_uint(pl.x) + (__float_as_uint(r.x) << 23));
  out.y = __uint_as_float(__float_as_uint(pl.y) + (__float_as_uint(r.y) << 23));
  return out;
}

// head_dim 128 tiling: key block width and S buffers per query tile (64 x 2 double-buffers S in TMEM)
#ifndef B200_BN128
#define B200_BN128 64
#endif
#ifndef B200_SB128
#define B200_SB128 2
#endif
#ifndef B200_POLY_OF_8
#define B200_POLY_OF_8 0
#endif
#ifndef B200_TAKE_TURNS
#define B200_TAKE_TURNS 0
#endif
// Of every 8 groups of 4 columns, this many have their exponentials evaluated on the FMA pipe.
constexpr int kPolyOf8 = B200_POLY_OF_8;
// Exp-phase turn-taking between the two query tiles of a CTA (tuning switch).
constexpr bool kTakeTurns = B200_TAKE_TURNS != 0;

// ---- one row (thread): its logits of a block in registers, COLS columns, masked outside [lo_c, hi_c] if MASK ----

// Maximum in base-2 units, -inf if every column is masked.  With a soft-cap the capped logit is a monotone function of the raw one, so
// the maximum is taken over the RAW values (no special-function work in this pass) and capped once; the pass also finds the largest
// |raw| so that the warp can vote for the polynomial-only exponential pass.
template <bool SOFTCAP, bool MASK, int COLS>
__device__ __forceinline__ float row_maximum(uint32_t (&sr)[COLS / 32][32], int lo_c, int hi_c, const FwdParams& p, float cmul,
                                             bool& cap_poly_only) {
  float mx0 = -INFINITY, mx1 = -INFINITY;
  [[maybe_unused]] float ab0 = 0.f, ab1 = 0.f;
#pragma unroll
  for (int ch = 0; ch < COLS / 32; ++ch) {
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      float v[4];
      [[maybe_unused]] float va[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float s = __uint_as_float(sr[ch][i + u]);
        [[maybe_unused]] float sa = s;
        if constexpr (MASK) {
          const int col = ch * 32 + i + u;
          if (col > hi_c || col < lo_c) {
            s = -INFINITY;
            sa = 0.f;
          }
          // (with a soft-cap the registers keep the raw value: the exponential pass masks by column again)
          if constexpr (!SOFTCAP) sr[ch][i + u] = __float_as_uint(s);
        }
        v[u] = s;
        if constexpr (SOFTCAP) va[u] = sa;
      }
      mx0 = fmax3(mx0, v[0], v[1]);
      mx1 = fmax3(mx1, v[2], v[3]);
      if constexpr (SOFTCAP) {
        ab0 = fmax3_abs(ab0, va[0], va[1]);
        ab1 = fmax3_abs(ab1, va[2], va[3]);
      }
    }
  }
  const float mx = fmaxf(mx0, mx1);
  if constexpr (SOFTCAP) {
    cap_poly_only = !__any_sync(0xffffffffu, fmaxf(ab0, ab1) * p.cap_in > kCapPolyMax);
    return mx == -INFINITY ? -INFINITY : softcap_tanh(mx * p.cap_in) * cmul;   // cap_out is folded into cmul
  } else {
    return mx * cmul;
  }
}

// P = exp2(x - m), packed to the 16-bit input type, written to TMEM from column p_addr on; returns the sum in fp32.
// POLY_ONLY: every |raw / cap| of the warp's columns is <= 1.
template <bool BF16, bool SOFTCAP, bool MASK, int COLS, bool POLY_ONLY>
__device__ __forceinline__ float row_exponentials_pass(const uint32_t (&sr)[COLS / 32][32], uint32_t p_addr, int lo_c, int hi_c,
                                                       const FwdParams& p, float cmul, float m) {
  const float2 c2 = make_float2(cmul, cmul), nm2 = make_float2(-m, -m);
  float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
  for (int ch = 0; ch < COLS / 32; ++ch) {
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      // x = logit - m in base-2 units for four columns
      float2 x0, x1;
      const float2 s0 = make_float2(__uint_as_float(sr[ch][i + 0]), __uint_as_float(sr[ch][i + 1]));
      const float2 s1 = make_float2(__uint_as_float(sr[ch][i + 2]), __uint_as_float(sr[ch][i + 3]));
      if constexpr (SOFTCAP) {
        const float2 a2 = make_float2(p.cap_in, p.cap_in);
        const float2 y0 = fmul2(s0, a2), y1 = fmul2(s1, a2);
        if constexpr (POLY_ONLY) {
          x0 = ffma2(y0, softcap_r2(y0, cmul), nm2);
          x1 = ffma2(y1, softcap_r2(y1, cmul), nm2);
        } else {
          x0 = ffma2(make_float2(softcap_tanh(y0.x), softcap_tanh(y0.y)), c2, nm2);
          x1 = ffma2(make_float2(softcap_tanh(y1.x), softcap_tanh(y1.y)), c2, nm2);
        }
        if constexpr (MASK) {
          const int col = ch * 32 + i;
          if (col + 0 > hi_c || col + 0 < lo_c) x0.x = -INFINITY;
          if (col + 1 > hi_c || col + 1 < lo_c) x0.y = -INFINITY;
          if (col + 2 > hi_c || col + 2 < lo_c) x1.x = -INFINITY;
          if (col + 3 > hi_c || col + 3 < lo_c) x1.y = -INFINITY;
        }
      } else {
        x0 = ffma2(s0, c2, nm2);
        x1 = ffma2(s1, c2, nm2);
      }
      // masked blocks hold -inf entries and stay on the special-function unit; elsewhere a fixed, interleaved
      // subset of the column groups goes through the polynomial
      if (!MASK && (((i / 4) * kPolyOf8) % 8) < kPolyOf8) {
        x0 = exp2_poly2(x0);
        x1 = exp2_poly2(x1);
      } else {
        x0.x = ex2_approx(x0.x);
        x0.y = ex2_approx(x0.y);
        x1.x = ex2_approx(x1.x);
        x1.y = ex2_approx(x1.y);
      }
      acc0 = fadd2(acc0, x0);
      acc1 = fadd2(acc1, x1);
      pk[i / 2] = pack2<BF16>(x0.x, x0.y);
      pk[i / 2 + 1] = pack2<BF16>(x1.x, x1.y);
    }
    tmem_st16(p_addr + ch * 16, pk);
  }
  return (acc0.x + acc0.y) + (acc1.x + acc1.y);
}
template <bool BF16, bool SOFTCAP, bool MASK, int COLS>
__device__ __forceinline__ float row_exponentials(const uint32_t (&sr)[COLS / 32][32], uint32_t p_addr, int lo_c, int hi_c,
                                                  const FwdParams& p, float cmul, float m, bool cap_poly_only) {
  if constexpr (SOFTCAP) {
    if (cap_poly_only) return row_exponentials_pass<BF16, SOFTCAP, MASK, COLS, true>(sr, p_addr, lo_c, hi_c, p, cmul, m);
  }
  return row_exponentials_pass<BF16, SOFTCAP, MASK, COLS, false>(sr, p_addr, lo_c, hi_c, p, cmul, m);
}

// O *= alpha for DIMS columns of the row's accumulator.
template <int DIMS>
__device__ __forceinline__ void row_rescale(uint32_t o_addr, float alpha) {
  const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
  for (int ch = 0; ch < DIMS / 16; ++ch) {
    uint32_t o[16];
    tmem_ld16(o_addr + ch * 16, o);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const float2 r = fmul2(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), a2);
      o[i] = __float_as_uint(r.x);
      o[i + 1] = __float_as_uint(r.y);
    }
    tmem_st16(o_addr + ch * 16, o);
  }
}

// O / l -> 16-bit -> global for DIMS columns of the row, from element `first` of `out` on (in_range: the row exists).
template <bool BF16, int DIMS>
__device__ __forceinline__ void row_store(uint32_t o_addr, void* out, int64_t first, float l, bool in_range) {
  const float inv_l = 1.0f / l;
  const bool wide_stores = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  uint4* out_row = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + first);
#pragma unroll
  for (int ch = 0; ch < DIMS / 32; ++ch) {
    uint32_t o[32];
    tmem_ld32(o_addr + ch * 32, o);
    tmem_ld_wait();
    if (in_range) {
      // every lane writes its own row (rows are heads * D elements apart), so a store instruction costs one
      // memory transaction per lane whatever its width: 32-byte stores halve the count
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          w[e] = pack2<BF16>(__uint_as_float(o[v * 16 + 2 * e]) * inv_l, __uint_as_float(o[v * 16 + 2 * e + 1]) * inv_l);
        if (wide_stores) {
          st_global_v8(out_row + ch * 4 + v * 2, w);
        } else {
          out_row[ch * 4 + v * 2] = make_uint4(w[0], w[1], w[2], w[3]);
          out_row[ch * 4 + v * 2 + 1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
  }
}

// One block of the online softmax for one row (thread).  MASK selects the edge-block variant.
template <class Cfg, bool BF16, bool SOFTCAP, bool MASK>
__device__ __forceinline__ bool fwd_softmax_block(const FwdCtx<Cfg, BF16>& c, const FwdParams& p, uint32_t s_addr,
                                                  uint32_t o_addr, uint64_t* o_full, uint64_t* p_full, int n,
                                                  int g, int lo_c, int hi_c, float cmul, float& m, float& l,
                                                  uint64_t* turn_wait, int turn_parity, uint64_t* turn_pass) {
  constexpr int D = Cfg::D, BN = Cfg::BN;
  const int lane = threadIdx.x & 31;
  // (tuning builds stamp the first 64 blocks a CTA walks)
  [[maybe_unused]] const int tl_base = (((int)(threadIdx.x >> 7)) * 64 + (g & 63)) * 8;
  [[maybe_unused]] const bool tl_on = (threadIdx.x & 127) == 0 && g < 64;
  if (tl_on) B200_TL(tl_base + 0);
  uint32_t sr[BN / 32][32];
#pragma unroll
  for (int ch = 0; ch < BN / 32; ++ch) tmem_ld32(s_addr + ch * 32, sr[ch]);
  tmem_ld_wait();
  if (tl_on) B200_TL(tl_base + 1);

  bool cap_poly_only = false;
  const float m_blk = row_maximum<SOFTCAP, MASK, BN>(sr, lo_c, hi_c, p, cmul, cap_poly_only);
  if (tl_on) B200_TL(tl_base + 2);
  float alpha = 1.0f;
  bool rescale = false;
  if (n == 0) {
    m = fmaxf(m, m_blk);
  } else if (m_blk - m > 8.0f) {
    // Lazy rescale: the running reference only moves when the new maximum exceeds it by more than 2^8, so
    // that exp2(x - m) stays <= 256 and the O accumulator is touched rarely.
    alpha = ex2_approx(m - m_blk);
    m = m_blk;
    l *= alpha;
    rescale = true;
  }
  if (n > 0 && __any_sync(0xffffffffu, rescale)) {
    // P V(n-1): barrier (n-1) % 2, phase (n-1) / 2.  S(n) has completed, hence every earlier MMA of this tile up to
    // P V(n-2) too, and P V(n+1) cannot start before this thread delivers P(n): the barrier is exactly in or
    // just past the awaited phase.
    // (g counts the P V products of this CTA: equal to n unless the CTA walks several tiles)
    if (!mbar_wait_warp(o_full + ((g - 1) & 1), ((g - 1) >> 1) & 1, c.abort_flag, WAIT_O_FULL)) return false;
    tc_fence_after();
    row_rescale<D>(o_addr, alpha);
  }
  // The exponentials saturate the special-function unit, which the warp of the other query tile on this SM
  // sub-partition shares: the two take turns (see fwd_softmax), so that one tile's exponentials overlap the
  // other tile's MMAs instead of colliding with its exponentials.
  if (turn_wait != nullptr && !mbar_wait_warp(turn_wait, turn_parity, c.abort_flag, WAIT_TURN)) return false;
  // P over the first BN/2 columns of S
  l += row_exponentials<BF16, SOFTCAP, MASK, BN>(sr, s_addr, lo_c, hi_c, p, cmul, m, cap_poly_only);
  if (turn_pass != nullptr) {
    __syncwarp();
    if (lane == 0) mbar_arrive(turn_pass);
  }
  if (tl_on) B200_TL(tl_base + 3);
  tmem_st_wait();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(p_full);
  if (tl_on) B200_TL(tl_base + 4);
  return true;
}

template <class Cfg, bool BF16, bool SOFTCAP>
__device__ __forceinline__ void fwd_softmax(const FwdCtx<Cfg, BF16>& c, const FwdParams& p, int t) {
  constexpr int D = Cfg::D, BN = Cfg::BN;
  const int warp_q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const TileRange rng = c.rng[t];
  if (rng.hi <= rng.lo) return;
  const int r_tile = c.q0 + t * Cfg::BM;
  const int row = r_tile + warp_q * 32 + lane;
  const uint32_t lane_addr = c.tmem_base + ((uint32_t)(warp_q * 32) << 16);
  constexpr int SB = Cfg::SB;
  const uint32_t s_addr0 = lane_addr + t * SB * BN;
  const uint32_t o_addr = lane_addr + Cfg::O_BASE + t * D;
  uint64_t* o_full = &c.bars[Cfg::BAR_O_FULL + t * 2];   // [2], P V(n) completes o_full[n % 2], phase n / 2

  const float cmul = SOFTCAP ? p.cap_out : p.scale_log2;
  float m = -1.0e30f;  // running reference maximum (base-2 units); finite so that fully masked blocks stay NaN-free
  float l = 0.f;
  // visible keys of this row: [lo_key, hi_key]
  const int hi_key = p.causal ? min(row + p.delta, p.kv_len - 1) : p.kv_len - 1;
  const int lo_key = (p.causal && p.window > 0) ? (row + p.delta - p.window + 1) : -(1 << 28);
  const int hi_first = p.causal ? min(r_tile + p.delta, p.kv_len - 1) : p.kv_len - 1;          // first row of the tile
  const int lo_last = (p.causal && p.window > 0) ? (r_tile + 127 + p.delta - p.window + 1) : -(1 << 28);  // last row

  // Turn-taking of the exponential phases between warp w of tile 0 and warp w of tile 1 (same SM sub-partition):
  // tile 0 runs its i-th phase after tile 1's (i-1)-th, tile 1 its i-th after tile 0's i-th.  A tile only waits
  // for phases the other tile really has (their block counts differ under a causal mask).
  uint64_t* turn_mine = nullptr;
  uint64_t* turn_other = nullptr;
  int n_other = 0;
  if constexpr (Cfg::NQ == 2 && kTakeTurns) {
    turn_mine = &c.bars[Cfg::BAR_TURN + t * 4 + warp_q];
    turn_other = &c.bars[Cfg::BAR_TURN + (1 - t) * 4 + warp_q];
    n_other = c.rng[1 - t].hi - c.rng[1 - t].lo;
  }

  for (int j = rng.lo; j < rng.hi; ++j) {
    const int n = j - rng.lo, buf = n % SB;
    const uint32_t s_addr = s_addr0 + buf * BN;
    uint64_t* p_full = &c.bars[Cfg::BAR_P_FULL + t * SB + buf];
    if (!mbar_wait_warp(&c.bars[Cfg::BAR_S_FULL + t * SB + buf], (n / SB) & 1, c.abort_flag, WAIT_S_FULL)) return;
    tc_fence_after();
    // a block needs element masks only if some row of the tile sees it partially
    const bool need_mask = (hi_first - j * BN < BN - 1) || (lo_last - j * BN > 0);
    uint64_t* tw = nullptr;
    int tpar = 0;
    if constexpr (Cfg::NQ == 2 && kTakeTurns) {
      const int need = (t == 0) ? n - 1 : n;          // index of the other tile's phase that must be over
      if (need >= 0 && need < n_other) {
        tw = turn_mine;
        tpar = need & 1;
      }
    }
    bool ok;
    if (need_mask)
      ok = fwd_softmax_block<Cfg, BF16, SOFTCAP, true>(c, p, s_addr, o_addr, o_full, p_full, n, n, lo_key - j * BN,
                                                       hi_key - j * BN, cmul, m, l, tw, tpar, turn_other);
    else
      ok = fwd_softmax_block<Cfg, BF16, SOFTCAP, false>(c, p, s_addr, o_addr, o_full, p_full, n, n, 0, 0, cmul, m, l, tw,
                                                        tpar, turn_other);
    if (!ok) return;
  }

  // epilogue: O / l -> 16-bit -> global (BSHD), base-2 LSE for the score passes
  if ((threadIdx.x & 127) == 0) B200_TL((3 * 64 + 62) * 8 + 2);   // last block's P delivered
  const int last = rng.hi - rng.lo - 1;
  if (!mbar_wait_warp(o_full + (last & 1), (last >> 1) & 1, c.abort_flag, WAIT_O_FULL)) return;
  tc_fence_after();
  if ((threadIdx.x & 127) == 0) B200_TL((3 * 64 + 62) * 8 + 3);   // last P V complete
  const bool in_range = row < p.q_len;
  row_store<BF16, D>(o_addr, p.out, (((int64_t)c.b * p.q_len + row) * p.heads + c.h) * (int64_t)D, l, in_range);
  if ((threadIdx.x & 127) == 0) B200_TL((3 * 64 + 62) * 8 + 4);   // output stored
  if (p.lse != nullptr && in_range) p.lse[((int64_t)c.b * p.heads + c.h) * p.lse_stride + row] = m + log2f(l);
}

// ----------------------------------- kernel ----------------------------------
template <int BN, int NQ, int SB, bool BF16, bool SOFTCAP>
__global__ void __launch_bounds__(FwdCfg<BN, NQ, SB>::THREADS, FwdCfg<BN, NQ, SB>::CTAS_PER_SM)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  using Cfg = FwdCfg<BN, NQ, SB>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);

  // A launch that follows an expired wait on this device drains immediately (the status word stays
  // set until the host reads it), so that one stuck kernel cannot stall a whole queue of launches.
  __shared__ int s_skip;
  if (threadIdx.x == 32) prefetch_l2(&g_device_status);   // read after the wait below
  [[maybe_unused]] const uint64_t cta_start_ns = global_timer_ns();
  [[maybe_unused]] const long long cta_start_clk = clock64();
  B200_TL_INIT();
  if (threadIdx.x == 0) B200_TL((3 * 64 + 62) * 8 + 0);   // kernel entry

  FwdCtx<Cfg, BF16> c;
  c.sQ = smem;
  c.sKV = c.sQ + NQ * Cfg::Q_TILE_BYTES;
  c.bars = reinterpret_cast<uint64_t*>(c.sKV + Cfg::SLOTS * Cfg::KV_STAGE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(c.bars + Cfg::NUM_BARS);
  c.abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heaviest query groups (largest row index => most visible key blocks) are scheduled first
  const int qg = gridDim.x - 1 - blockIdx.x;
  c.q0 = qg * Cfg::BM * NQ;
  c.h = blockIdx.y;
  c.b = blockIdx.z;
  c.hk = c.h / (p.heads / p.kv_heads);
  c.jmin = 1 << 30;
  c.jmax = 0;
#pragma unroll
  for (int t = 0; t < NQ; ++t) {
    c.rng[t] = tile_range(c.q0 + t * Cfg::BM, BN, p);
    if (c.rng[t].hi > c.rng[t].lo) {
      c.jmin = min(c.jmin, c.rng[t].lo);
      c.jmax = max(c.jmax, c.rng[t].hi);
    }
  }
  if (c.jmax == 0) c.jmin = 0;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < Cfg::NUM_BARS; ++i) {
      const bool is_p_full = (i >= Cfg::BAR_P_FULL && i < Cfg::BAR_P_FULL + NQ * SB);          // 4 softmax warps
      const bool is_empty = (i >= Cfg::BAR_EMPTY && i < Cfg::BAR_EMPTY + Cfg::SLOTS);           // NQ MMA issuers
      mbar_init(&c.bars[i], is_p_full ? 4u : is_empty ? (uint32_t)NQ : 1u);
    }
    *c.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == NQ * 4 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  // The wait comes before the TMEM allocation and the status word: a predecessor that let this launch start early may still have
  // to allocate columns of its own, and what it wrote is visible only now.
  pdl_wait();
  if (threadIdx.x == 32) s_skip = *reinterpret_cast<volatile int*>(&g_device_status);
  if (warp == 0) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem_base = *tmem_slot;
  if (s_skip != 0) {
    if (warp == 0) tmem_dealloc(c.tmem_base, Cfg::TMEM_COLS);
    return;
  }
  if (threadIdx.x == 0) B200_TL((3 * 64 + 62) * 8 + 1);   // set-up done (barriers, TMEM)

  if (warp < NQ * 4) {
    if constexpr (Cfg::REBALANCE_REGS) reg_alloc<224>();
    if constexpr (NQ == 2) {
      // the tile index is a compile-time constant inside each branch (no dynamic indexing of per-tile state)
      if (warp < 4)
        fwd_softmax<Cfg, BF16, SOFTCAP>(c, p, 0);
      else
        fwd_softmax<Cfg, BF16, SOFTCAP>(c, p, 1);
    } else {
      fwd_softmax<Cfg, BF16, SOFTCAP>(c, p, 0);
    }
  } else {
    if constexpr (Cfg::REBALANCE_REGS) reg_dealloc<56>();
    if (warp == NQ * 4) {
      if (lane == 0) fwd_producer<Cfg, BF16>(c, &tm_q, &tm_k, &tm_v);
    } else if (warp == NQ * 4 + 1) {
      fwd_mma<Cfg, BF16, 0>(c);
    } else if (NQ == 2 && warp == NQ * 4 + 2) {
      fwd_mma<Cfg, BF16, NQ - 1>(c);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) B200_TL((3 * 64 + 62) * 8 + 5);   // all roles done
  if (warp == 0) tmem_dealloc(c.tmem_base, Cfg::TMEM_COLS);
  B200_TL_FLUSH();
  B200_TL_CTA(cta_start_ns, cta_start_clk, c.jmax - c.jmin);
}

// --------------------------------- host side ---------------------------------
template <int BN, int NQ, int SB, bool BF16, bool SOFTCAP>
int launch_attn_fwd_cfg(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p,
                        cudaStream_t stream) {
  using Cfg = FwdCfg<BN, NQ, SB>;
  auto kern = attn_fwd_kernel<BN, NQ, SB, BF16, SOFTCAP>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  B200_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    configured_dev = dev;
  }
  const int groups = (p.q_len + Cfg::BM * NQ - 1) / (Cfg::BM * NQ);
  dim3 grid(groups, p.heads, p.batch);
  B200_CUDA_TRY(launch_kernel(kern, grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream, 1, tq, tk, tv, p));
  return B200_OK;
}

// persistent variant (attn_fwd_persist.cuh)
template <bool BF16, bool SOFTCAP>
int launch_attn_fwd_persist(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
                            const FwdParams& p, cudaStream_t stream);

// head_dim 256 (attn_fwd_split.cuh)
struct AttnStrides;
template <bool BF16, bool SOFTCAP>
int launch_attn_fwd_split(const void* q, const void* k, const void* v, const FwdParams& p, const AttnStrides& st,
                          bool one_tile_per_cta, cudaStream_t stream);

// element strides of q / k / v when they are views into a larger buffer (0 = contiguous)
struct AttnStrides {
  int64_t q_token, q_batch, k_token, k_batch, v_token, v_batch;
};

// few query rows against many keys (attn_decode.cuh)
bool use_decode(int q_len, int group);
int attn_decode_impl(const void* q, const void* k, const void* v, const FwdParams& f, int head_dim, bool bf16,
                     const AttnStrides& st, cudaStream_t stream);

inline int attn_fwd_impl_lse_stride(const void* q, const void* k, const void* v, void* out, float* lse,
                                    int lse_stride, int batch, int q_len, int kv_len, int heads, int kv_heads,
                                    int head_dim, int dtype, int causal, int window, float softcap, float scale,
                                    cudaStream_t stream, const AttnStrides* strides = nullptr) {
  if (!q || !k || !v || !out) return B200_ERR_BAD_ARGUMENT;
  if (batch <= 0 || q_len <= 0 || kv_len <= 0 || heads <= 0 || kv_heads <= 0) return B200_ERR_BAD_ARGUMENT;
  if (dtype != B200_F16 && dtype != B200_BF16) return B200_ERR_BAD_DTYPE;
  if (head_dim != 128 && head_dim != 256) return B200_ERR_UNSUPPORTED;
  if (heads % kv_heads != 0) return B200_ERR_BAD_ARGUMENT;
  if (kv_len < q_len) return B200_ERR_UNSUPPORTED;  // rows without any visible key (the reference yields NaN)
  if (window > 0 && !causal) return B200_ERR_UNSUPPORTED;
  if (!(scale > 0.f) || softcap < 0.f) return B200_ERR_BAD_ARGUMENT;
  if (heads > 65535 || batch > 65535) return B200_ERR_UNSUPPORTED;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out)) return B200_ERR_MISALIGNED;

  const bool bf16 = dtype == B200_BF16;
  const AttnStrides contiguous{0, 0, 0, 0, 0, 0};
  const AttnStrides& st = strides ? *strides : contiguous;
  FwdParams p;
  p.out = out;
  p.lse = lse;
  p.lse_stride = lse_stride;
  p.batch = batch;
  p.q_len = q_len;
  p.kv_len = kv_len;
  p.heads = heads;
  p.kv_heads = kv_heads;
  p.causal = causal ? 1 : 0;
  p.window = window > 0 ? window : 0;
  p.delta = kv_len - q_len;
  const float kLog2e = 1.4426950408889634f;
  p.scale_log2 = scale * kLog2e;
  p.cap_in = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_out = softcap * kLog2e;
  if (use_decode(q_len, heads / kv_heads)) return attn_decode_impl(q, k, v, p, head_dim, bf16, st, stream);

  const bool cap = softcap > 0.f;
  // The grids are persistent; a launch of one CTA per tile stays selectable for A/B timing (read once per process).
  static const bool one_tile_per_cta = std::getenv("B200_ATTN_ONE_TILE_PER_CTA") != nullptr;
  if (head_dim == 256) {
    return bf16 ? (cap ? launch_attn_fwd_split<true, true>(q, k, v, p, st, one_tile_per_cta, stream)
                       : launch_attn_fwd_split<true, false>(q, k, v, p, st, one_tile_per_cta, stream))
                : (cap ? launch_attn_fwd_split<false, true>(q, k, v, p, st, one_tile_per_cta, stream)
                       : launch_attn_fwd_split<false, false>(q, k, v, p, st, one_tile_per_cta, stream));
  }

  const int bn = B200_BN128;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tensor_map(&tq, q, batch, q_len, heads, head_dim, 128, bf16, st.q_token, st.q_batch)) != B200_OK)
    return rc;
  if ((rc = make_bshd_tensor_map(&tk, k, batch, kv_len, kv_heads, head_dim, bn, bf16, st.k_token, st.k_batch)) != B200_OK)
    return rc;
  if ((rc = make_bshd_tensor_map(&tv, v, batch, kv_len, kv_heads, head_dim, bn, bf16, st.v_token, st.v_batch)) != B200_OK)
    return rc;

  // Default: the persistent kernel, whose CTAs walk query tiles handed out by an atomic counter, two CTAs per SM.  (The other
  // kernel also supports NQ = 2 -- two tiles sharing one K/V stream in a single CTA; two independent CTAs per SM measured 13 %
  // faster at seq 4096.)
#ifdef B200_NQ128
  constexpr int NQ = B200_NQ128;
#else
  constexpr int NQ = 1;
#endif
  if (!one_tile_per_cta && B200_BN128 == 64 && B200_SB128 == 2) {
    CUtensorMap to = tq;   // a warp stores 32 rows (unused with a soft-cap)
    if (!cap && (rc = make_bshd_tensor_map(&to, out, batch, q_len, heads, head_dim, 32, bf16)) != B200_OK) return rc;
    return bf16 ? (cap ? launch_attn_fwd_persist<true, true>(tq, tk, tv, to, p, stream)
                       : launch_attn_fwd_persist<true, false>(tq, tk, tv, to, p, stream))
                : (cap ? launch_attn_fwd_persist<false, true>(tq, tk, tv, to, p, stream)
                       : launch_attn_fwd_persist<false, false>(tq, tk, tv, to, p, stream));
  }
  return bf16 ? (cap ? launch_attn_fwd_cfg<B200_BN128, NQ, B200_SB128, true, true>(tq, tk, tv, p, stream)
                     : launch_attn_fwd_cfg<B200_BN128, NQ, B200_SB128, true, false>(tq, tk, tv, p, stream))
              : (cap ? launch_attn_fwd_cfg<B200_BN128, NQ, B200_SB128, false, true>(tq, tk, tv, p, stream)
                     : launch_attn_fwd_cfg<B200_BN128, NQ, B200_SB128, false, false>(tq, tk, tv, p, stream));
}

inline int attn_fwd_impl(const void* q, const void* k, const void* v, void* out, float* lse, int batch, int q_len,
                         int kv_len, int heads, int kv_heads, int head_dim, int dtype, int causal, int window,
                         float softcap, float scale, cudaStream_t stream) {
  return attn_fwd_impl_lse_stride(q, k, v, out, lse, q_len, batch, q_len, kv_len, heads, kv_heads, head_dim, dtype,
                                  causal, window, softcap, scale, stream);
}

}  // namespace b200
