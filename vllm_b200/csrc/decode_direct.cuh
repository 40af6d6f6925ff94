// Decode attention for batches that are bound by latency, not by bandwidth: few (sequence, kv head)
// pairs, or short sequences.
//
// The persistent kernel (decode_kernel.cuh) is built to keep HBM busy; a launch with little work pays
// for that with a long chain: prefix plan of the whole batch, shared-memory ring, one page after the
// other in each warp, partials through global memory, arrival counters, one warp merging dozens of
// partials.  Here a (sequence, kv head, head group) belongs to one CLUSTER of 1 to 16 CTAs of four
// warps:
//   * its 16-token tiles are dealt to all warps of the cluster in contiguous ranges, so that a warp has
//     one to a few of them;
//   * K and V go from global memory straight into the registers that mma.sync reads (a warp load
//     covers whole 128- to 256-byte runs of a page): no ring, no barriers, the next tile's K and V are
//     requested as soon as this one's have been consumed;
//   * the order of tokens inside a tile and of head dimensions inside the QK product is permuted so
//     that a lane's 16 bytes of a page (8 bytes of V) are its operand registers as they come;
//   * the warps' partials are merged in shared memory, those of the CTAs through distributed shared
//     memory, all in fp32: two cluster barriers instead of global counters.
// Measured on B200 against the persistent kernel, see direct_plan in paged_attention.cu.
#pragma once

#include <type_traits>

#include "decode_kernel.cuh"

namespace b200pa {

constexpr int kDirectWarps = 4;

__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_stream8(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_stream4(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of this CTA's shared-memory location `addr` in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster16(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_cluster8(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

template <int KV, int D, int GP>
struct DirectShape {
  static constexpr int kHeads = 8 * GP;
  static constexpr int kRow = D + 4;  // floats between two heads: spreads a warp's stores over the banks
  static constexpr int kSmem = kDirectWarps * kHeads * kRow * 4;
  // registers of one tile of K and V, of the accumulators and Q
  static constexpr int kTileRegs = D / (KV != kCache16 ? 4 : 2);
  static constexpr int kOtherRegs = 3 * D * GP / 8;
  // tiles in flight per warp, and resident CTAs per SM that the register budget is set for
  static constexpr int kBufs = 2 * kTileRegs + kOtherRegs <= 120 ? 2 : 1;
  static constexpr int kMinCtas = kBufs * kTileRegs + kOtherRegs <= 128 ? 3 : 2;
  // CTAs that fit (head size 32 and one head tile needs 117 registers, everything else more than 128)
  static constexpr int kResident = D == 32 && GP == 1 ? 4 : kMinCtas;
};

// grid.x = (sequence, kv head, head group) items x cluster size.
template <typename QT, int KV, int D, int GP>
__global__ void __launch_bounds__(kDirectWarps * 32, DirectShape<KV, D, GP>::kMinCtas)
pa_decode_direct_kernel(const DecodeParams p, const int cluster) {
  using TR = DecodeTraits<QT, KV, D, GP>;
  using SH = DirectShape<KV, D, GP>;
  constexpr bool kFp8 = TR::kFp8;
  constexpr bool kBf = TR::kMmaBf16;
  constexpr bool kE5 = KV == kCacheE5M2;
  constexpr bool kOutBf = std::is_same_v<QT, __nv_bfloat16>;
  constexpr int ES = TR::kEsize;
  constexpr int X = 16 / ES;                   // head dimensions per 16-byte chunk of K
  constexpr int CHUNKS = D / X;                // ... chunks per token
  constexpr int NI = (CHUNKS + 3) / 4;         // chunks per lane (lane c takes chunks c, c + 4, ...)
  constexpr int SPC = X / 4;                   // MMA k-steps that a lane's chunk feeds
  constexpr int KS = (D + 15) / 16;            // d tiles of the P.V product
  constexpr int HEADS = SH::kHeads;
  constexpr int ROW = SH::kRow;
  extern __shared__ __align__(16) float s_part[];  // [warp][head][ROW]: partial outputs
  __shared__ float2 s_ml[kDirectWarps][HEADS];     // (max logit, exp sum) of the warps
  __shared__ float2 s_cta[HEADS];                  // ... of the CTA

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, c = lane & 3;
  const int rank = cluster == 1 ? 0 : int(cluster_rank());
  int item = int(blockIdx.x) / cluster;
  const int hg = item % p.head_groups;
  item /= p.head_groups;
  const int kvh = item % p.num_kv_heads;
  const int seq = item / p.num_kv_heads;
  const int hq0 = kvh * p.group + hg * HEADS;
  const int nheads = min(HEADS, p.group - hg * HEADS);
  const int B = p.block_size, b_shift = 31 - __clz(B);
  if (!p.early) grid_dependency();

  const int len = min(max(__ldcg(p.seq_lens + seq), 0), p.len_cap);
  // ---- Q (B operand; n = head g): 16 bytes of K's chunk order per chunk of this lane
  uint32_t qf[GP][NI][SPC][2];
#pragma unroll
  for (int nt = 0; nt < GP; ++nt) {
    const int hl = nt * 8 + g;
    const QT* q = static_cast<const QT*>(p.q) + int64_t(seq) * p.q_stride + int64_t(hq0 + hl) * D;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int ch = 4 * i + c;
      uint32_t w[X / 2];
      const bool ok = hl < nheads && (CHUNKS % 4 == 0 || ch < CHUNKS);
#pragma unroll
      for (int k = 0; k < X / 8; ++k) {
        const uint4 v = ok ? __ldcg(reinterpret_cast<const uint4*>(q + ch * X) + k) : make_uint4(0, 0, 0, 0);
        w[4 * k] = v.x;
        w[4 * k + 1] = v.y;
        w[4 * k + 2] = v.z;
        w[4 * k + 3] = v.w;
      }
      if constexpr (kFp8 && kOutBf) {  // operands of an fp8 cache are f16
#pragma unroll
        for (int k = 0; k < X / 2; ++k)
          w[k] = pack2<false>(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u));
      }
#pragma unroll
      for (int s = 0; s < SPC; ++s) {
        qf[nt][i][s][0] = w[2 * s];
        qf[nt][i][s][1] = w[2 * s + 1];
      }
    }
  }
  const float qk_scale = p.scale * kLog2e * (kFp8 ? __ldcg(p.k_scale) : 1.f);
  float slope[GP][2];
#pragma unroll
  for (int nt = 0; nt < GP; ++nt)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int hl = nt * 8 + 2 * c + j;
      slope[nt][j] = (p.alibi != nullptr && hl < nheads) ? __ldcg(p.alibi + hq0 + hl) * kLog2e : 0.f;
    }

  // ---- this warp's 16-token tiles [t_begin, t_end)
  const int tiles = (len + 15) >> 4;
  const int nw = cluster * kDirectWarps, gw = rank * kDirectWarps + warp;
  const int t_begin = int(int64_t(tiles) * gw / nw), t_end = int(int64_t(tiles) * (gw + 1) / nw);
  const int* bt = p.block_tables + int64_t(seq) * p.max_blocks_per_seq;
  const char* kb = static_cast<const char*>(p.kc) + int64_t(kvh) * p.kv_head_stride * ES;
  const char* vb = static_cast<const char*>(p.vc) + int64_t(kvh) * p.kv_head_stride * ES;
  const int64_t bstride = p.kv_block_stride * ES;
  int ids = 0;
  auto load_ids = [&](int t0) {  // block ids of tiles t0 .. t0 + 31
    ids = t0 + lane < t_end ? __ldcg(bt + (((t0 + lane) << 4) >> b_shift)) : 0;
  };
  // row rho = 8 h + g of the tile's S^T is token 4 (g / 2) + 2 h + g % 2: a lane's V tokens 4c .. 4c+3
  // are then the k indices that its registers of the P.V product stand for
  const int tok_g = 4 * (g >> 1) + (g & 1);
  constexpr int NB = SH::kBufs;
  uint4 kr[NB][NI][2];
  using VWord = std::conditional_t<kFp8, uint32_t, uint2>;
  VWord vr[NB][KS][2];
  auto get_k = [&](int t, uint4 (&kr)[NI][2]) {
    const int64_t blk = __shfl_sync(0xffffffffu, ids, (t - t_begin) & 31);
    const char* src = kb + blk * bstride + ((t << 4) & (B - 1)) * 16 + tok_g * 16;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int ch = 4 * i + c;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        kr[i][h] = (CHUNKS % 4 == 0 || ch < CHUNKS) ? ld_stream16(src + int64_t(ch * B + 2 * h) * 16)
                                                    : make_uint4(0, 0, 0, 0);
    }
  };
  auto get_v = [&](int t, VWord (&vr)[KS][2]) {
    const int64_t blk = __shfl_sync(0xffffffffu, ids, (t - t_begin) & 31);
    const char* src = vb + blk * bstride + (((t << 4) & (B - 1)) + 4 * c) * ES;
#pragma unroll
    for (int mt = 0; mt < KS; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int d = 16 * mt + 8 * h + g;
        if constexpr (kFp8) vr[mt][h] = ld_stream4(src + d * B);
        else vr[mt][h] = (16 * mt + 8 * h < D) ? ld_stream8(src + d * B * 2) : make_uint2(0, 0);
      }
  };

  float o[KS][GP][4];
#pragma unroll
  for (int mt = 0; mt < KS; ++mt)
#pragma unroll
    for (int nt = 0; nt < GP; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[mt][nt][i] = 0.f;
  float m_run[GP][2], l_run[GP][2];
#pragma unroll
  for (int nt = 0; nt < GP; ++nt) {
    m_run[nt][0] = m_run[nt][1] = -INFINITY;
    l_run[nt][0] = l_run[nt][1] = 0.f;
  }
  if (t_begin < t_end) load_ids(t_begin);
  if (p.early) grid_dependency();  // (from here on K and V)
  if (t_begin < t_end) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (t_begin + b < t_end) {
        get_k(t_begin + b, kr[b]);
        get_v(t_begin + b, vr[b]);
      }
    }
  }
  // tile t, whose K and V are in (or on their way to) kr and vr; they are requested for tile t + NB
  // as soon as the registers are free
  auto step = [&](int t, uint4 (&kr)[NI][2], VWord (&vr)[KS][2]) {
    const int tok0 = t << 4;
    // ---- S^T = K . Q^T (two accumulation chains)
    float s[GP][4], s2[GP][4];
#pragma unroll
    for (int nt = 0; nt < GP; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[nt][i] = s2[nt][i] = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      uint32_t a[2][X / 2];  // rows g and g + 8: the chunk as operand words
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t raw[4] = {kr[i][h].x, kr[i][h].y, kr[i][h].z, kr[i][h].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if constexpr (kFp8) fp8x4_to_f16<kE5>(raw[k], a[h][2 * k], a[h][2 * k + 1]);
          else a[h][k] = raw[k];
        }
      }
#pragma unroll
      for (int st = 0; st < SPC; ++st)
#pragma unroll
        for (int nt = 0; nt < GP; ++nt)
          mma16816<kBf>((st & 1) ? s2[nt] : s[nt], a[0][2 * st], a[1][2 * st], a[0][2 * st + 1],
                        a[1][2 * st + 1], qf[nt][i][st][0], qf[nt][i][st][1]);
    }
    if (t + NB < t_end) {
      if (((t + NB - t_begin) & 31) == 0) load_ids(t + NB);
      get_k(t + NB, kr);
    }
    // ---- online softmax
    const bool need_mask = tok0 + 16 > len;
    const int tok_lo = tok0 + tok_g, tok_hi = tok_lo + 2;
    float alpha[GP][2];
#pragma unroll
    for (int nt = 0; nt < GP; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float lo = (s[nt][j] + s2[nt][j]) * qk_scale, hi = (s[nt][2 + j] + s2[nt][2 + j]) * qk_scale;
        if (p.alibi != nullptr) {
          lo += slope[nt][j] * float(tok_lo - len + 1);
          hi += slope[nt][j] * float(tok_hi - len + 1);
        }
        if (need_mask) {
          if (tok_lo >= len) lo = -INFINITY;
          if (tok_hi >= len) hi = -INFINITY;
        }
        float mx = fmaxf(lo, hi);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        mx = fmaxf(mx, m_run[nt][j]);  // finite: every tile holds at least one valid token
        alpha[nt][j] = fast_exp2(m_run[nt][j] - mx);
        m_run[nt][j] = mx;
        s[nt][j] = fast_exp2(lo - mx);
        s[nt][2 + j] = fast_exp2(hi - mx);
        l_run[nt][j] = l_run[nt][j] * alpha[nt][j] + (s[nt][j] + s[nt][2 + j]);
      }
    if (t > t_begin) {
#pragma unroll
      for (int mt = 0; mt < KS; ++mt)
#pragma unroll
        for (int nt = 0; nt < GP; ++nt) {
          o[mt][nt][0] *= alpha[nt][0];
          o[mt][nt][1] *= alpha[nt][1];
          o[mt][nt][2] *= alpha[nt][0];
          o[mt][nt][3] *= alpha[nt][1];
        }
    }
    // ---- O^T += V^T . P^T
    uint32_t pf[GP][2];
#pragma unroll
    for (int nt = 0; nt < GP; ++nt) {
      pf[nt][0] = movm_trans(pack2<kBf>(s[nt][0], s[nt][1]));
      pf[nt][1] = movm_trans(pack2<kBf>(s[nt][2], s[nt][3]));
    }
    if (need_mask) {  // stale bytes behind the end could be NaN: V of those tokens becomes zero
      const int left = len - (tok0 + 4 * c);  // valid ones of this lane's four tokens
#pragma unroll
      for (int mt = 0; mt < KS; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if constexpr (kFp8) {
            vr[mt][h] = left >= 4 ? vr[mt][h] : (left <= 0 ? 0u : vr[mt][h] & (0xffffffffu >> (32 - 8 * left)));
          } else {
            if (left < 2) vr[mt][h].x = left <= 0 ? 0u : vr[mt][h].x & 0xffffu;
            if (left < 4) vr[mt][h].y = left <= 2 ? 0u : vr[mt][h].y & 0xffffu;
          }
        }
    }
#pragma unroll
    for (int mt = 0; mt < KS; ++mt) {
      uint32_t a0, a1, a2, a3;
      if constexpr (kFp8) {
        fp8x4_to_f16<kE5>(vr[mt][0], a0, a2);
        fp8x4_to_f16<kE5>(vr[mt][1], a1, a3);
      } else {
        a0 = vr[mt][0].x;
        a2 = vr[mt][0].y;
        a1 = vr[mt][1].x;
        a3 = vr[mt][1].y;
      }
#pragma unroll
      for (int nt = 0; nt < GP; ++nt) mma16816<kBf>(o[mt][nt], a0, a1, a2, a3, pf[nt][0], pf[nt][1]);
    }
    if (t + NB < t_end) get_v(t + NB, vr);
  };
  for (int t = t_begin; t < t_end; t += NB) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (b == 0 || t + b < t_end) step(t + b, kr[b], vr[b]);
  }

  // ---- the warp's partial: (m, l) per head, O relative to m
  float* mine = s_part + warp * HEADS * ROW;
#pragma unroll
  for (int nt = 0; nt < GP; ++nt)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float l = l_run[nt][j];
      l += __shfl_xor_sync(0xffffffffu, l, 4);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      const int hl = nt * 8 + 2 * c + j;
      if (g == 0) s_ml[warp][hl] = make_float2(m_run[nt][j], l);
      if (hl < nheads && t_begin < t_end) {
#pragma unroll
        for (int mt = 0; mt < KS; ++mt) {
          mine[hl * ROW + 16 * mt + g] = o[mt][nt][j];
          if (16 * mt + 8 < D) mine[hl * ROW + 16 * mt + 8 + g] = o[mt][nt][2 + j];
        }
      }
    }
  __syncthreads();

  // ---- merges.  A unit is four head dimensions of one head.
  constexpr int UPH = D / 4;
  const float kv_o = kFp8 ? *p.v_scale : 1.f;
  auto store = [&](int hl, int d, float4 acc, float m, float l) {
    const float inv = kv_o * __fdividef(1.f, l + 1e-6f);
    uint2 w;
    w.x = pack2<kOutBf>(acc.x * inv, acc.y * inv);
    w.y = pack2<kOutBf>(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(static_cast<QT*>(p.out) + (int64_t(seq) * p.num_heads + hq0 + hl) * D + d) = w;
    if (p.lse != nullptr && d == 0)
      p.lse[int64_t(hq0 + hl) * p.num_seqs + seq] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
  };
  // the four warps
  for (int u = tid; u < nheads * UPH; u += kDirectWarps * 32) {
    const int hl = u / UPH, d = (u % UPH) * 4;
    float2 ml[kDirectWarps];
    float m = -INFINITY, l = 0.f;
#pragma unroll
    for (int w = 0; w < kDirectWarps; ++w) {
      ml[w] = s_ml[w][hl];
      m = fmaxf(m, ml[w].x);
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kDirectWarps; ++w) {
      if (ml[w].y > 0.f) {  // (a warp without tiles has written no output)
        const float f = fast_exp2(ml[w].x - m);
        l += ml[w].y * f;
        const float4 v = *reinterpret_cast<const float4*>(s_part + (w * HEADS + hl) * ROW + d);
        acc.x += f * v.x;
        acc.y += f * v.y;
        acc.z += f * v.z;
        acc.w += f * v.w;
      }
    }
    if (cluster == 1) {
      store(hl, d, acc, m, l);
    } else {
      *reinterpret_cast<float4*>(s_part + hl * ROW + d) = acc;  // (this thread's unit only)
      if (d == 0) s_cta[hl] = make_float2(m, l);
    }
  }
  if (cluster == 1) return;
  // the CTAs: each takes its share of the units of all of them
  cluster_arrive();
  cluster_wait();
  const uint32_t part0 = smem_u32(s_part), cta0 = smem_u32(s_cta);
  for (int u = rank * kDirectWarps * 32 + tid; u < nheads * UPH; u += cluster * kDirectWarps * 32) {
    const int hl = u / UPH, d = (u % UPH) * 4;
    float m = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r0 = 0; r0 < cluster; r0 += 8) {  // eight CTAs' values requested at a time
      float2 ml[8];
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool ok = r0 + k < cluster;
        const uint32_t r = ok ? r0 + k : 0;
        ml[k] = ld_cluster8(cluster_map(cta0 + hl * 8, r));
        v[k] = ld_cluster16(cluster_map(part0 + (hl * ROW + d) * 4, r));
        if (!ok) ml[k] = make_float2(-INFINITY, 0.f);
      }
      float m_new = m;
#pragma unroll
      for (int k = 0; k < 8; ++k) m_new = fmaxf(m_new, ml[k].x);
      const float old = m_new == -INFINITY ? 0.f : fast_exp2(m - m_new);
      l *= old;
      acc = make_float4(acc.x * old, acc.y * old, acc.z * old, acc.w * old);
      m = m_new;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (ml[k].y > 0.f) {
          const float f = fast_exp2(ml[k].x - m);
          l += ml[k].y * f;
          acc.x += f * v[k].x;
          acc.y += f * v[k].y;
          acc.z += f * v[k].z;
          acc.w += f * v[k].w;
        }
      }
    }
    store(hl, d, acc, m, l);
  }
  cluster_arrive();  // nobody leaves while its shared memory may be read
  cluster_wait();
}

}  // namespace b200pa
