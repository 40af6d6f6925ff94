// Large KV writes of 16-bit key/value tensors (prefill steps): tiles of 16 tokens by tensor map, one
// slot look-up per tile instead of one per tile, head and half.
//
// What bounds it: HBM, once the instructions per element are few.  The staged kernel (kv_write_staged.cuh)
// spends 16 a bf16 element on a quantising write, 9 of them on its work items (16 tokens of one head of K or
// V, each with its own slot look-up, window search and 16 row copies); here
//   * a work item is 16 tokens x 2 heads of K and V, fetched with one tensor-map box per 64 head dimensions
//     (128-byte swizzle) into a ring of three stages, four CTAs to an SM (4 heads and two CTAs: 1 to 12 % more
//     below 10000 tokens; 1 head and eight: up to 13 % less below, 3 % more on the largest);
//   * one warp walks over the tiles: slots, window (see below), copies; four warps convert, half a head of
//     K and of V each (V takes longer, so not K in four of them and V in the others), with all loops
//     unrolled and the head size a constant;
//   * K (and V of the flash layout): a lane converts 16 bytes of output of one token; V of the x-layout: the
//     transpose by ldmatrix.trans as in the staged kernel.
// Windows (x-layout): a row of V there holds the tokens of one block, so a tile writes whole words of it only
// if its tokens lie in slots as they lie in the tile.  A tile whose first, ninth and last slots are
// consecutive modulo 16 covers the 16 tokens from the next 16-slot boundary on instead of its own, those of
// the next tile only if that one is moved as far; what it gives up in front is a second window, which ends at
// that boundary, unless the tile before is moved as far.  Three slots of a tile decide, the same for it and
// for its neighbours; whatever the slots are, every token is written, with its own slot.
// Measured on B200, staged kernel -> this one, us: 128 chunks of 128 tokens that start anywhere, 8 heads of
// 128, to fp8 36.4 -> 23.5 (4.3 TB/s), 16 bit 43 -> 29.8; 32 chunks of 100 to 160, fp8, 15.1 -> 10.0; flash
// layout 16384 tokens, fp8, 21.9 -> 20.1.  What is left over 15.6 of traffic: start and end, about 6, and 10
// instructions an element.
#pragma once

#include <cuda.h>

#include "kv_write_staged.cuh"
#include "kv_write_windows.h"
#include "tcgen05.cuh"

namespace b200pa {

struct TileWriteParams {
  void* key_cache;
  void* value_cache;
  const int64_t* slot_mapping;
  const float* k_scale;
  const float* v_scale;
  int* status;
  int64_t block_stride;  // flash layout: elements of the cache
  int64_t page_stride;
  int64_t head_stride;
  int num_tokens;
  int num_heads;         // a multiple of kTileHeads
  int block_size;
};

constexpr int kTileHeads = 2;                     // heads per item
constexpr int kTileStages = 3;
constexpr int kTileThreads = (2 * kTileHeads + 1) * 32;

template <int D>
struct TileShape {
  static constexpr int kBoxes = D / 64;
  static constexpr int kBoxBytes = kTileHeads * 16 * 128;       // [head][token][64 elements]
  static constexpr int kStage = 2 * kBoxes * kBoxBytes;         // K's boxes, then V's
  static constexpr int kSmem = 1024 + kTileStages * kStage;     // (1024: alignment)
  static constexpr int kCtas = D <= 128 ? 4 : 2;                // per SM
  static_assert(D % 64 == 0 && kCtas * (kSmem + 1536) <= 227 * 1024, "shared memory");
};

template <typename in_t, typename cache_t, int KV, int D, bool kFlash>
__global__ void __launch_bounds__(kTileThreads, TileShape<D>::kCtas)
kv_write_tiles_kernel(const TileWriteParams p, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
  using SH = TileShape<D>;
  constexpr int E = sizeof(cache_t), NST = kTileStages, W = 2 * kTileHeads;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t s_bar[2 * NST];
  __shared__ __align__(16) int64_t s_slot[NST][16];
  __shared__ int s_head[NST];  // first head of the item, < 0: no more items
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar0 = smem_u32(s_bar);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (NST + s); };
  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), W);
    }
    fence_barrier_init();
  }
  __syncthreads();
  grid_dependency();

  const int H = p.num_heads, B = p.block_size, N = p.num_tokens;
  const int b_shift = 31 - __clz(B);  // a power of two
  auto give_up = [&] {
    if (lane == 0) atomicExch(p.status, kStatusMbarTimeout);
  };
  int stage = 0;
  uint32_t round = 0;
  auto next_stage = [&] {
    if (++stage == NST) {
      stage = 0;
      ++round;
    }
  };

  if (warp == W) {
    // ================================================= slots, windows, copies
    const int tiles = (N + 15) / 16, groups = H / kTileHeads, items = tiles * groups;
    auto slot_at = [&](int tok) -> int64_t { return tok >= 0 && tok < N ? __ldg(p.slot_mapping + tok) : int64_t(-1); };
    // Lanes 0 .. 15: the tile's slots, 16 .. 31: those of the next one; and in lanes 0 .. 2 the first, ninth and
    // last of the one before.  Requested an item ahead.
    auto look = [&](int item) -> int64_t { return item < items ? slot_at(item % tiles * 16 + lane) : int64_t(-1); };
    auto look_back = [&](int item) -> int64_t {
      return item < items && lane < 3 ? slot_at(item % tiles * 16 - 16 + (lane == 0 ? 0 : (lane == 1 ? 8 : 15))) : int64_t(-1);
    };
    auto from = [&](int64_t v, int l) { return __shfl_sync(0xffffffffu, v, l); };
    bool ok = true;
    // one window: tokens from `tok` on, of which rows lo .. hi - 1 are to be written; `slot` is row lane's
    auto put = [&](int tok, int lo, int hi, int head0, int64_t slot) {
      if (round > 0 && !__all_sync(0xffffffffu, mbar_wait(empty(stage), (round - 1) & 1))) {
        ok = false;
        return;
      }
      if (lane < 16) s_slot[stage][lane] = lane >= lo && lane < hi ? slot : int64_t(-1);
      if (lane == 0) s_head[stage] = head0;
      __syncwarp();
      if (lane == 0) {
        mbar_expect_tx(full(stage), SH::kStage);
#pragma unroll
        for (int x = 0; x < SH::kBoxes; ++x) {
          tma_load3(smem + stage * SH::kStage + x * SH::kBoxBytes, &kmap, x * 64, tok, head0, full(stage));
          tma_load3(smem + stage * SH::kStage + (SH::kBoxes + x) * SH::kBoxBytes, &vmap, x * 64, tok, head0, full(stage));
        }
      }
      __syncwarp();
      next_stage();
    };
    // Neighbouring tiles of the same heads to a CTA: tiles with two windows, or with a run's end in them, are
    // spread over the CTAs so; a stride of the grid may meet all of them.
    const int begin = int(int64_t(items) * blockIdx.x / gridDim.x), end = int(int64_t(items) * (blockIdx.x + 1) / gridDim.x);
    int64_t cand = look(begin), cand_back = look_back(begin);
    for (int item = begin; item < end && ok; ++item) {
      const int64_t now = cand, back = cand_back;
      if (item + 1 < end) {
        cand = look(item + 1);
        cand_back = look_back(item + 1);
      }
      const int t0 = item % tiles * 16, head0 = item / tiles * kTileHeads;
      int d = 0, before = 0, after = 0;
      if (!kFlash) {
        d = tile_shift(from(now, 0), from(now, 8), from(now, 15));
        before = tile_shift(from(back, 0), from(back, 1), from(back, 2));
        after = tile_shift(from(now, 16), from(now, 24), from(now, 31));
      }
      const TileWindow own = tile_window(t0, N, d, after), front = tile_front_window(t0, d, before);
      put(own.tok, own.lo, own.hi, head0, from(now, (lane + d) & 31));
      // (at a negative or a foreign token the box starts with rows that nobody writes)
      if (ok && front.lo < front.hi) put(front.tok, front.lo, front.hi, head0, from(now, (lane + d) & 15));
    }
    // the end; then nobody leaves with copies on their way
    if (ok && round > 0) ok = __all_sync(0xffffffffu, mbar_wait(empty(stage), (round - 1) & 1));
    if (ok) {
      if (lane == 0) {
        s_head[stage] = -1;
        mbar_arrive(full(stage));
      }
      __syncwarp();
    } else {
      give_up();
      for (int i = 0; i < NST; ++i) {  // stages that were filled in this round, or in the one before
        const uint32_t r = i < stage ? round : round - 1;
        if (i < stage || round > 0) mbar_wait(full(i), r & 1);
      }
    }
    return;
  }

  // ================================================= conversion: half a head of K and of V
  const int hl = warp >> 1, part = warp & 1;
  const ScaledDiv k_div(KV == kKvAuto ? 1.f : *p.k_scale), v_div(KV == kKvAuto ? 1.f : *p.v_scale);
  for (;; next_stage()) {
    if (!__all_sync(0xffffffffu, mbar_wait(full(stage), round & 1))) {
      give_up();
      return;
    }
    const int h = s_head[stage] + hl;
    if (s_head[stage] < 0) return;
    // ---- a token to a lane, 16-byte chunks of cache: even ones by lanes 0 .. 15, odd ones by the others
    auto rows = [&](uint32_t src, void* cache, const ScaledDiv& div) {
      const int t = lane & 15, odd = lane >> 4;
      const int64_t slot = s_slot[stage][t];
      const int64_t blk = slot >> b_shift;
      const int off = int(slot) & (B - 1);
      constexpr int CH = 16 / E, NCH = D / CH;  // elements of a chunk, chunks
      unsigned char* dst = static_cast<unsigned char*>(cache);
      int64_t step;  // bytes between two chunks of a token
      if constexpr (kFlash) {
        dst += (blk * p.block_stride + int64_t(off) * p.page_stride + int64_t(h) * p.head_stride) * E;
        step = 16;
      } else {
        dst += ((blk * H + h) * int64_t(NCH) * B + off) * 16;
        step = int64_t(B) * 16;
      }
      dst += (part * (NCH / 2) + odd) * step;
      if (slot >= 0) {
        const uint32_t row = src + t * 128;
#pragma unroll
        for (int i = 0; i < NCH / 4; ++i) {
          // chunk 2 i + odd of this half; its 16 bytes (fp8: two of them) of the row, swizzled
          constexpr int PB = 64 / CH;  // chunks per box
          const int c = part * (NCH / 2) + 2 * i;
          const uint32_t at = row + c / PB * SH::kBoxBytes;
          const int q = KV == kKvAuto ? (c % PB + odd) ^ (t & 7) : ((c % PB + odd) * 2) ^ (t & 7);
          const uint4 a = ld_shared16(at + q * 16);
          uint4 out = a;
          if constexpr (KV != kKvAuto) {
            const uint4 b = ld_shared16(at + (q ^ 1) * 16);
            const uint32_t wi[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            uint32_t wo[4];
            convert_words<in_t, KV, 8>(wi, wo, div);
            out = make_uint4(wo[0], wo[1], wo[2], wo[3]);
          }
          *reinterpret_cast<uint4*>(dst + 2 * i * step) = out;
        }
      }
    };
    const uint32_t k_src = smem + stage * SH::kStage + hl * (16 * 128);
    const uint32_t v_src = k_src + SH::kBoxes * SH::kBoxBytes;
    rows(k_src, p.key_cache, k_div);
    if constexpr (kFlash) {
      rows(v_src, p.value_cache, v_div);
    } else {
      // ---- V of the x-layout (kv_write_staged.cuh explains the matrices): lane j = lane % 4 gets tokens
      // 4 j .. 4 j + 3 of rows d = lane / 4 and 8 more
      const int j = lane & 3;
      int64_t sl[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) sl[k] = s_slot[stage][4 * j + k];
      const bool quad = sl[0] >= 0 && (sl[0] & 3) == 0 && sl[1] == sl[0] + 1 && sl[2] == sl[0] + 2 && sl[3] == sl[0] + 3;
      auto place = [&](int64_t s) {  // of a slot's element of this lane's first row
        return static_cast<cache_t*>(p.value_cache) + (((s >> b_shift) * H + h) * D + part * (D / 2) + (lane >> 2)) * int64_t(B) +
               (s & (B - 1));
      };
      const int mr = lane & 7, mi = lane >> 3;
      const int mtok = (mr >> 1) * 4 + (mr & 1) + (mi & 1) * 2;
      const uint32_t row = v_src + mtok * 128, chunk = uint32_t((mi >> 1) ^ (mtok & 7)) * 16;
      auto pass = [&](auto exact_tag) -> uint32_t {
        constexpr bool kExact = decltype(exact_tag)::value;
        (void)kExact;
        uint32_t nan_bits = 0;
        cache_t* dst = place(sl[0]);
#pragma unroll
        for (int i16 = 0; i16 < D / 32; ++i16) {
          const int d16 = part * (D / 32) + i16;
          uint32_t r[4];  // (tokens 4j, 4j+1), (4j+2, 4j+3) of row d; the same of row d + 8
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                       : "r"(row + d16 / 4 * SH::kBoxBytes + (chunk ^ (d16 % 4 * 32))));
          uint32_t w[2][2];  // this lane's piece of row d and of row d + 8 (one word when fp8)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if constexpr (KV == kKvAuto) {
              w[i][0] = r[2 * i];
              w[i][1] = r[2 * i + 1];
            } else if constexpr (kExact) {
              const uint32_t in[2] = {r[2 * i], r[2 * i + 1]};
              uint32_t o[1];
              convert_words<in_t, KV, 2>(in, o, v_div);  // (checks its own codes)
              w[i][0] = o[0];
            } else {
              const uint32_t v = neg_quant4<in_t, KV == kKvE5M2>(r[2 * i], r[2 * i + 1], v_div);
              nan_bits |= (v & 0x7F7F7F7Fu) + 0x01010101u;
              w[i][0] = v ^ 0x80808080u;
            }
          }
          const int64_t o = int64_t(i16) * 16 * B;
          if (quad) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if constexpr (E == 1) *reinterpret_cast<uint32_t*>(dst + o + 8 * i * B) = w[i][0];
              else *reinterpret_cast<uint2*>(dst + o + 8 * i * B) = make_uint2(w[i][0], w[i][1]);
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (sl[k] < 0) continue;
              cache_t* one = place(sl[k]) + o;
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                if constexpr (E == 1) *reinterpret_cast<unsigned char*>(one + 8 * i * B) = static_cast<unsigned char>(w[i][0] >> (8 * k));
                else *reinterpret_cast<uint16_t*>(one + 8 * i * B) = static_cast<uint16_t>(w[i][k >> 1] >> (16 * (k & 1)));
              }
            }
          }
        }
        return nan_bits & 0x80808080u;
      };
      if constexpr (KV == kKvAuto) {
        pass(std::false_type{});
      } else {
        // (ldmatrix is warp-collective: the decision to repeat with the division is taken by the warp)
        const bool again = !v_div.fast || __any_sync(0xffffffffu, pass(std::false_type{}) != 0);
        if (again) pass(std::true_type{});
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty(stage));
  }
}

}  // namespace b200pa
