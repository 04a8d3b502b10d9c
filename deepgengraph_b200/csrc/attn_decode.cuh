// Attention forward for a handful of query rows against a long key range (generation steps: q_len 1, or a few tokens,
// against a K/V cache):  out = softmax(mask(softcap(q k^T * scale))) v.
//
// The work is the read of K and V (2 FLOP per byte and query row), so the kernel is laid out for bytes in flight, not for
// the tensor pipe:
//   * the group * q_len query rows that share a K/V head (at most 16) are ONE tile, so every K/V element is read once
//     -- the 128-row kernel reads it once per query head and walks the keys of a head in one serial chain of 64-key blocks;
//   * a unit (batch, K/V head) is split over a cluster of CTAs (attn_decode_plan.h) that merge through distributed shared
//     memory: no scratch, no second launch, no atomics;
//   * inside a CTA the warps take 16-key tiles in turn, each with its own ring of three stages filled by 16-byte cp.async:
//     no CTA-wide barrier until the merge, 128 KB in flight per SM;
//   * the products are mma.sync m16n8k16: a tcgen05 tile would be 128 rows high for 1 to 16 rows of use, and the
//     contraction needs 5 % of what even mma.sync delivers.
// Measured (bf16, head_dim 128, GPU time): batch 8, 32 query / 8 K/V heads, 8192 keys 115.6 -> 42 us (6.4 TB/s; 96 % of the
// copy rate with the launch gap); batch 4, 32 heads, 512 keys 11.0 -> 7.0 us.
// The 16-bit rounding of P, the fp32 accumulation and the base-2 log-sum-exp are those of the tile kernel.
#pragma once

#include "attn_decode_plan.h"
#include "attn_fwd.cuh"

namespace b200 {

constexpr int kDecodeRows = 16;     // query rows of a unit that one CTA takes (the M of the MMA)
constexpr int kDecodeStages = 3;

struct DecodeParams {
  const uint16_t *q, *k, *v;
  uint16_t* out;
  float* lse;
  int lse_stride;
  int q_len, kv_len, heads, kv_heads, group;
  int64_t q_token, q_batch, k_token, k_batch, v_token, v_batch;   // strides in elements
  int causal, window, delta;
  float scale_log2, cap_in, cap_out;
  int first_tile, n_tiles, tiles_per_cta;   // 16-key tiles that hold at least one visible key, and a CTA's share
};

template <int D, int WARPS_>
struct DecodeCfg {
  static constexpr int WARPS = WARPS_;
  static constexpr int TILE_BYTES = 16 * D * 2;                      // 16 keys of K or V
  static constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  static constexpr int RING_BYTES = WARPS * kDecodeStages * STAGE_BYTES;
  static constexpr int O_PITCH = D + 8;                              // floats; rows of the partial outputs
  static_assert(WARPS * kDecodeRows * O_PITCH * 4 <= RING_BYTES, "partial outputs reuse the ring");
  static constexpr int SMEM_BYTES = RING_BYTES + 2 * (WARPS + 1) * kDecodeRows * 4;
  static constexpr int CTAS_PER_SM = SMEM_BYTES <= 113 * 1024 ? 2 : 1;
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool pred) {
  const int n = pred ? 16 : 0;   // 0 source bytes: the destination is zero-filled
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// d (16 x 8, fp32) += a (16 x 16) * b (16 x 8)
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_map(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

template <int D, int WARPS, bool BF16, bool SOFTCAP>
__global__ void __launch_bounds__(WARPS * 32, (DecodeCfg<D, WARPS>::CTAS_PER_SM)) attn_decode_kernel(const DecodeParams p) {
  using Cfg = DecodeCfg<D, WARPS>;
  constexpr int KK = D / 16;           // k steps of Q K^T
  constexpr int CH = D / 8;            // 16-byte chunks of a row
  extern __shared__ __align__(128) uint8_t smem[];
  float* s_m = reinterpret_cast<float*>(smem + Cfg::RING_BYTES);   // [warps + 1][16] row maxima; the last row is the CTA's
  float* s_l = s_m + (WARPS + 1) * kDecodeRows;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.x, rank = blockIdx.y, n_ranks = gridDim.y;
  const int b = unit / p.kv_heads, hk = unit - b * p.kv_heads;
  const int rows = p.q_len * p.group;
  const uint16_t* k_head = p.k + b * p.k_batch + (int64_t)hk * D;
  const uint16_t* v_head = p.v + b * p.v_batch + (int64_t)hk * D;
  const int t_lo = p.first_tile + rank * p.tiles_per_cta;
  const int t_hi = min(t_lo + p.tiles_per_cta, p.first_tile + p.n_tiles);
  pdl_wait();

  // ---- this warp's ring: tile t of the warp goes to stage t % 3; rows of D * 2 bytes, 16-byte chunk c of row r at c ^ (r & 7)
  const uint32_t ring = smem_u32(smem) + warp * (kDecodeStages * Cfg::STAGE_BYTES);
  auto load_tile = [&](int tile, int stage) {
    const uint32_t dst = ring + stage * Cfg::STAGE_BYTES;
#pragma unroll
    for (int it = 0; it < CH / 2; ++it) {
      const int id = it * 32 + lane, r = id / CH, c = id % CH;
      const int key = tile * 16 + r;
      const bool in = key < p.kv_len;
      const int64_t row = in ? key : 0;
      const uint32_t off = r * (D * 2) + ((c ^ (r & 7)) << 4);
      cp_async_16(dst + off, k_head + row * p.k_token + c * 8, in);
      cp_async_16(dst + Cfg::TILE_BYTES + off, v_head + row * p.v_token + c * 8, in);
    }
  };
  int next = t_lo + warp;
#pragma unroll
  for (int s = 0; s < kDecodeStages - 1; ++s) {
    if (next < t_hi) load_tile(next, s);
    cp_async_commit();
    next += WARPS;
  }

  // ---- Q fragments: row i of the tile is query i / group, head hk * group + i % group
  const int row0 = lane >> 2, row1 = row0 + 8;
  auto q_row = [&](int i) -> const uint16_t* {
    const int qi = i / p.group, g = i - qi * p.group;
    return p.q + b * p.q_batch + (int64_t)qi * p.q_token + (int64_t)(hk * p.group + g) * D;
  };
  uint32_t qf[KK][4];
  {
    const bool in0 = row0 < rows, in1 = row1 < rows;
    const uint32_t* q0 = reinterpret_cast<const uint32_t*>(q_row(in0 ? row0 : 0)) + (lane & 3);
    const uint32_t* q1 = reinterpret_cast<const uint32_t*>(q_row(in1 ? row1 : 0)) + (lane & 3);
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
      qf[kk][0] = in0 ? q0[kk * 8] : 0u;
      qf[kk][1] = in1 ? q1[kk * 8] : 0u;
      qf[kk][2] = in0 ? q0[kk * 8 + 4] : 0u;
      qf[kk][3] = in1 ? q1[kk * 8 + 4] : 0u;
    }
  }
  // visible keys of the thread's two rows
  int hi_key[2], lo_key[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int pos = min(e == 0 ? row0 : row1, rows - 1) / p.group + p.delta;
    hi_key[e] = p.causal ? min(pos, p.kv_len - 1) : p.kv_len - 1;
    lo_key[e] = p.window > 0 ? pos - p.window + 1 : 0;
  }

  float o[CH][4];
#pragma unroll
  for (int j = 0; j < CH; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m[2] = {-1.0e30f, -1.0e30f}, l[2] = {0.f, 0.f};

  // ldmatrix lane roles: matrix mi = lane / 8, row lane % 8 of it.  K: key (mi / 2) * 8 + row, chunk 2 kk + (mi & 1);
  // V (transposed): key (mi & 1) * 8 + row, chunk 2 jj + mi / 2.  Both keys are congruent to lane % 8 modulo 8.
  const int mi = lane >> 3, sw = lane & 7;
  const uint32_t k_row = ((mi >> 1) * 8 + sw) * (D * 2), v_row = Cfg::TILE_BYTES + ((mi & 1) * 8 + sw) * (D * 2);
  int stage = 0;
  for (int tile = t_lo + warp; tile < t_hi; tile += WARPS) {
    cp_async_wait<kDecodeStages - 2>();
    __syncwarp();
    {   // the stage consumed in the previous iteration is free: every lane has passed the barrier above
      const int fill = stage == 0 ? kDecodeStages - 1 : stage - 1;
      if (next < t_hi) load_tile(next, fill);
      cp_async_commit();
      next += WARPS;
    }
    const uint32_t base = ring + stage * Cfg::STAGE_BYTES;
    float s[2][4] = {}, s_odd[2][4] = {};   // two accumulators: the MMAs of a chain wait for one another
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
      uint32_t kf[4];
      ldmatrix_x4(kf, base + k_row + (((2 * kk + (mi & 1)) ^ sw) << 4));
      mma_16816<BF16>((kk & 1) ? s_odd[0] : s[0], qf[kk], kf[0], kf[1]);
      mma_16816<BF16>((kk & 1) ? s_odd[1] : s[1], qf[kk], kf[2], kf[3]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e >> 2][e & 3] += s_odd[e >> 2][e & 3];
    const int key0 = tile * 16 + (lane & 3) * 2;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int key = key0 + nt * 8 + (e & 1), r = e >> 1;
        float x = SOFTCAP ? softcap_tanh(s[nt][e] * p.cap_in) * p.cap_out : s[nt][e] * p.scale_log2;
        if (key > hi_key[r] || key < lo_key[r]) x = -INFINITY;
        s[nt][e] = x;
        mx[r] = fmaxf(mx[r], x);
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    }
    if (__any_sync(0xffffffffu, mx[0] > m[0] || mx[1] > m[1])) {
      float a[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m_new = fmaxf(m[r], mx[r]);
        a[r] = ex2_approx(m[r] - m_new);
        m[r] = m_new;
        l[r] *= a[r];
      }
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        o[j][0] *= a[0];
        o[j][1] *= a[0];
        o[j][2] *= a[1];
        o[j][3] *= a[1];
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[nt][e] = ex2_approx(s[nt][e] - m[e >> 1]);
        l[e >> 1] += s[nt][e];
      }
    const uint32_t pf[4] = {pack2<BF16>(s[0][0], s[0][1]), pack2<BF16>(s[0][2], s[0][3]), pack2<BF16>(s[1][0], s[1][1]),
                            pack2<BF16>(s[1][2], s[1][3])};
#pragma unroll
    for (int jj = 0; jj < CH / 2; ++jj) {
      uint32_t vf[4];
      ldmatrix_x4_trans(vf, base + v_row + (((2 * jj + (mi >> 1)) ^ sw) << 4));
      mma_16816<BF16>(o[2 * jj], pf, vf[0], vf[1]);
      mma_16816<BF16>(o[2 * jj + 1], pf, vf[2], vf[3]);
    }
    stage = stage == kDecodeStages - 1 ? 0 : stage + 1;
  }

  // ---- merge of the CTA's warps (partial outputs in the ring's memory), then of the cluster's CTAs ----
  cp_async_wait<0>();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
  }
  __syncthreads();
  float* s_o = reinterpret_cast<float*>(smem);   // [warps][16][O_PITCH]
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = r == 0 ? row0 : row1;
    if (row < rows) {
      float* dst = s_o + (warp * kDecodeRows + row) * Cfg::O_PITCH + (lane & 3) * 2;
#pragma unroll
      for (int j = 0; j < CH; ++j) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
      if ((lane & 3) == 0) {
        s_m[warp * kDecodeRows + row] = m[r];
        s_l[warp * kDecodeRows + row] = l[r];
      }
    }
  }
  __syncthreads();
  auto store = [&](int row, int d, float4 acc, float m_row, float l_row) {
    const float inv = 1.0f / l_row;
    const int qi = row / p.group, h = hk * p.group + (row - qi * p.group);
    const uint2 w = make_uint2(pack2<BF16>(acc.x * inv, acc.y * inv), pack2<BF16>(acc.z * inv, acc.w * inv));
    *reinterpret_cast<uint2*>(p.out + (((int64_t)b * p.q_len + qi) * p.heads + h) * D + d) = w;
    if (d == 0 && p.lse != nullptr) p.lse[((int64_t)b * p.heads + h) * p.lse_stride + qi] = m_row + log2f(l_row);
  };
  const int n_vec = rows * (D / 4);
  for (int i = threadIdx.x; i < n_vec; i += WARPS * 32) {
    const int row = i / (D / 4), d = (i % (D / 4)) * 4;
    float mm = s_m[row];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) mm = fmaxf(mm, s_m[w * kDecodeRows + row]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float ll = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = ex2_approx(s_m[w * kDecodeRows + row] - mm);
      const float4 x = *reinterpret_cast<const float4*>(s_o + (w * kDecodeRows + row) * Cfg::O_PITCH + d);
      acc.x = fmaf(f, x.x, acc.x);
      acc.y = fmaf(f, x.y, acc.y);
      acc.z = fmaf(f, x.z, acc.z);
      acc.w = fmaf(f, x.w, acc.w);
      ll = fmaf(f, s_l[w * kDecodeRows + row], ll);
    }
    if (n_ranks == 1) {
      store(row, d, acc, mm, ll);
    } else {
      *reinterpret_cast<float4*>(s_o + row * Cfg::O_PITCH + d) = acc;   // only this thread reads or writes these elements
      if (d == 0) {
        s_m[WARPS * kDecodeRows + row] = mm;
        s_l[WARPS * kDecodeRows + row] = ll;
      }
    }
  }
  if (n_ranks == 1) return;
  cluster_arrive();
  cluster_wait();
  const uint32_t o_addr = smem_u32(s_o), m_addr = smem_u32(s_m + WARPS * kDecodeRows),
                 l_addr = smem_u32(s_l + WARPS * kDecodeRows);
  for (int i = rank * (WARPS * 32) + threadIdx.x; i < n_vec; i += n_ranks * (WARPS * 32)) {
    const int row = i / (D / 4), d = (i % (D / 4)) * 4;
    float mm = -INFINITY;
    for (int c = 0; c < n_ranks; ++c) mm = fmaxf(mm, ld_cluster(cluster_map(m_addr + row * 4, c)));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float ll = 0.f;
#pragma unroll 4
    for (int c = 0; c < n_ranks; ++c) {
      const float f = ex2_approx(ld_cluster(cluster_map(m_addr + row * 4, c)) - mm);
      const float4 x = ld_cluster4(cluster_map(o_addr + (row * Cfg::O_PITCH + d) * 4, c));
      acc.x = fmaf(f, x.x, acc.x);
      acc.y = fmaf(f, x.y, acc.y);
      acc.z = fmaf(f, x.z, acc.z);
      acc.w = fmaf(f, x.w, acc.w);
      ll = fmaf(f, ld_cluster(cluster_map(l_addr + row * 4, c)), ll);
    }
    store(row, d, acc, mm, ll);
  }
  cluster_arrive();   // the other CTAs may still be reading this one's shared memory
  cluster_wait();
}

// How many clusters of `c` CTAs of a kernel the device holds at once; 0 if it cannot hold any.
template <class Kernel>
inline int placeable_clusters(Kernel kern, int c, int threads, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = (unsigned)c;
  attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(1, c);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

template <int D, int WARPS, bool BF16, bool SOFTCAP>
int launch_attn_decode(DecodeParams p, int units, int c, cudaStream_t stream) {
  using Cfg = DecodeCfg<D, WARPS>;
  auto kern = attn_decode_kernel<D, WARPS, BF16, SOFTCAP>;
  static thread_local int configured_dev = -1, placeable = 0;   // of the largest clusters
  int dev = 0;
  B200_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    placeable = placeable_clusters(kern, kDecodeMaxCluster, WARPS * 32, Cfg::SMEM_BYTES);
    configured_dev = dev;
  }
  c = decode_cluster_that_fits(c, units, placeable);
  p.tiles_per_cta = (p.n_tiles + c - 1) / c;
  B200_CUDA_TRY(launch_kernel(kern, dim3(units, c), WARPS * 32, Cfg::SMEM_BYTES, stream, c, p));
  return B200_OK;
}

// Taken when the query rows of a unit fit one MMA tile: beyond that the 128-row tile kernel has enough rows to share a K/V
// block among.  A function of the unit alone: a shard of the heads or batch elements goes to the same kernel as the whole problem.
inline bool use_decode(int q_len, int group) { return (int64_t)q_len * group <= kDecodeRows; }

inline int attn_decode_impl(const void* q, const void* k, const void* v, const FwdParams& f, int head_dim, bool bf16,
                            const AttnStrides& st, cudaStream_t stream) {
  DecodeParams p;
  p.q = static_cast<const uint16_t*>(q);
  p.k = static_cast<const uint16_t*>(k);
  p.v = static_cast<const uint16_t*>(v);
  p.out = static_cast<uint16_t*>(f.out);
  p.lse = f.lse;
  p.lse_stride = f.lse_stride;
  p.q_len = f.q_len;
  p.kv_len = f.kv_len;
  p.heads = f.heads;
  p.kv_heads = f.kv_heads;
  p.group = f.heads / f.kv_heads;
  p.q_token = st.q_token ? st.q_token : (int64_t)f.heads * head_dim;
  p.k_token = st.k_token ? st.k_token : (int64_t)f.kv_heads * head_dim;
  p.v_token = st.v_token ? st.v_token : (int64_t)f.kv_heads * head_dim;
  p.q_batch = st.q_batch ? st.q_batch : p.q_token * f.q_len;
  p.k_batch = st.k_batch ? st.k_batch : p.k_token * f.kv_len;
  p.v_batch = st.v_batch ? st.v_batch : p.v_token * f.kv_len;
  p.causal = f.causal;
  p.window = f.causal ? f.window : 0;
  p.delta = f.delta;
  p.scale_log2 = f.scale_log2;
  p.cap_in = f.cap_in;
  p.cap_out = f.cap_out;
  const int first_key = p.window > 0 ? std::max(0, f.delta - p.window + 1) : 0;
  p.first_tile = first_key / 16;
  p.n_tiles = (f.kv_len + 15) / 16 - p.first_tile;
  p.tiles_per_cta = p.n_tiles;
  const bool cap = f.cap_out > 0.f;
  const int units = f.batch * f.kv_heads;
  const DecodeSplit split = decode_split(units, p.n_tiles, sm_count());
  const int c = split.ctas;
#define B200_DECODE_W(D_, W_)                                                                \
  (bf16 ? (cap ? launch_attn_decode<D_, W_, true, true>(p, units, c, stream)                  \
               : launch_attn_decode<D_, W_, true, false>(p, units, c, stream))                \
        : (cap ? launch_attn_decode<D_, W_, false, true>(p, units, c, stream)                 \
               : launch_attn_decode<D_, W_, false, false>(p, units, c, stream)))
  if (head_dim == 128) return split.wide ? B200_DECODE_W(128, 8) : B200_DECODE_W(128, 4);
  return split.wide ? B200_DECODE_W(256, 4) : B200_DECODE_W(256, 2);
#undef B200_DECODE_W
}

}  // namespace b200
