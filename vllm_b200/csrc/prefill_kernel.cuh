// Attention of query chunks (prefill, chunked prefill) over the paged cache, on the fifth-generation
// tensor cores.  Every request r of a step brings q_len tokens, the last q_len positions of its
// sequence; token i attends to the cached positions up to its own (causal).  The new tokens' K and V
// are in the cache already.
//
// What bounds it: the two contractions are 4 * D flops per (query head, query, key), so with a few
// hundred query rows per K/V tile the tensor cores and the exponentials are the limit, not HBM.
// The decode kernel reads the whole context once per query TOKEN; here a K/V tile is read once per
// 256 query rows.
//
//   * One persistent CTA per SM: two softmax warpgroups (one thread per query row), one
//     producer warpgroup for K and V, one warp that issues the MMAs, one that draws work items and
//     works out what they cover, one (two for fp8) that brings Q.
//   * A work item is (request, 2 x 128 query rows, kv head).  A row is one (token, query head of the
//     group): the heads that share a kv head are packed into the rows of a tile, so K/V are fetched
//     once for all of them, and the causal edge of a tile is only 128 / group tokens wide.
//   * S = Q.K^T and O += P.V are tcgen05.mma (M = 128, fp32 accumulators in TMEM).  K sits in shared
//     memory as [16-byte granule along D][key][16 bytes], the no-swizzle K-major operand layout, which the
//     x-layout of the K cache gives without any transposition; V as its pages lie, with 32-byte swizzle
//     (fp8 caches: widened, [8 keys][D][16 bytes]); Q as tensor-map boxes with swizzle.  P goes back to
//     TMEM as the A operand of the second product, over S.
//   * The two row tiles take turns: while the softmax of one runs, the tensor cores work for the
//     other.
//   * A thread takes its whole row of S into registers (one TMEM read, paired fp32 arithmetic,
//     three-way maxima; 528 -> 506 us before V and Q came by tensor map) and hands P over in two halves:
//     the product of the first runs under the exponentials of the second.  With an fp8 cache or a bias the
//     maximum of the tile comes before its first exponential; otherwise a row that has a maximum starts
//     with that one, and the tile is done again where it was too low (363 -> 353 us).
//   * The running maximum is only raised (and O rescaled in TMEM) when a row's maximum grew by more
//     than 2^8 to 2^12: until then P is merely larger than 1, which fp32 sums and 16-bit P hold as exactly.
//   * fp8 caches are widened to f16 (exact) by the producers on their way to shared memory.
//   * Few items (short chunks behind long contexts): the keys of an item are cut into pieces, every
//     piece leaves a normalised partial, and the warp that delivers the last piece of its rows merges
//     them.  Nobody waits for another CTA.
//   * Every mbarrier wait is bounded; on expiry a status code is recorded and all roles leave.
//
// Measured on B200, a step of 4 chunks (8192 tokens, contexts up to 4096, 32 / 8 heads of 128, bf16;
// KV write included): 8970 us with one decode work item per token, 346 us here (1160 TFLOP/s; 400 when it
// runs for long and the power limit holds the clock down).  Start to first product: 15000 cycles when every role worked an item out for itself and Q came with 16-byte copies, 9300
// now (3400 plan, 2200 item, 500 Q, K beside it), which is what steps of short chunks consist of: 20 to
// 35 us, 10 to 25 % less.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "decode_kernel.cuh"
#include "tcgen05.cuh"

namespace b200pa {

struct PrefillParams {
  void* out;                  // [num_tokens, num_heads, D]
  const void* q;              // [num_tokens, num_heads, D], token stride q_stride
  const void* kc;
  const void* vc;
  const int* block_tables;
  const int* seq_lens;        // per request, this step's tokens included
  const int* q_start;         // [num_reqs + 1]
  const float* alibi;
  const float* k_scale;
  const float* v_scale;
  unsigned* sched;            // [0] ticket, [1] CTAs done (self-resetting)
  unsigned* arrive;           // arrival counters of split row tiles
  unsigned char* ws;          // partials of split row tiles
  int* status;
  int64_t q_stride;
  int64_t kv_block_stride;    // elements
  int64_t kv_head_stride;
  int num_reqs;
  int num_tokens;
  int num_heads;
  int num_kv_heads;
  int group;
  int block_size;
  int max_blocks_per_seq;
  int ws_slots;               // pieces that the workspace has room for
  // What a kernel reads before its own wait has been written by grids that are complete (the one in front has
  // waited for them, and lets the next one in only then); copies by tensor map, which are another proxy's
  // accesses and which no wait of this grid stands in front of, are ordered behind it by a fence.
  int late_wait;              // 1: independent of the launch in front, waits for it at the end only
  int early;                  // 1: the launch in front is the step's KV write, see launch_dependent
  float scale;
};

constexpr int kPrefillThreads = 16 * 32;
// Registers per thread: 512 threads start with 128 each; the softmax warpgroups take over what the
// others give back.  (The producers of an fp8 cache hold a K and a V tile in registers.  An 8192-token
// fp8 step of 64 / 8 heads takes 1032 us with 176 / 112 / 48 and 997 with 184 / 104 / 40.)
template <bool kFp8>
struct PrefillRegs {
  static constexpr int kSoftmax = kFp8 ? 184 : 192, kProducer = kFp8 ? 104 : 80, kMma = kFp8 ? 40 : 48;
  static_assert(2 * kSoftmax + kProducer + kMma == 4 * 128, "register split");
};
constexpr int kPrefillMaxReqs = 512;    // requests per launch: prefix table in shared memory
constexpr int kPrefillSortReqs = 64;    // up to so many are taken longest first (the reason is with the plan)

template <int D>
struct PrefillShape {
  static constexpr int DP = (D + 15) / 16 * 16;     // operand width (head size 120 is padded)
  static constexpr int NQ = D > 192 ? 1 : 2;        // row tiles per item: TMEM holds NQ * (KT + DP) columns
  static constexpr int KT = D > 128 ? 64 : 128;     // keys per tile
  static constexpr int kQBytes = 128 * DP * 2;
  static constexpr int kTileBytes = KT * DP * 2;
  // ring of K and V tiles in turns (K0, V0, K1, V1, ...): what shared memory holds besides Q
  static constexpr int kRoom = 223 * 1024 - NQ * kQBytes;
  static constexpr int kSlots = kRoom / kTileBytes < 8 ? kRoom / kTileBytes : 8;
  static constexpr int kSmem = NQ * kQBytes + kSlots * kTileBytes;
  // Q comes in boxes of 64 head dimensions (128-byte swizzle) where the head size allows, else of 16
  static constexpr int kQBox = D % 64 == 0 ? 64 : 16;
  static_assert(kSlots >= 4, "a K and a V tile in use, another of each on its way");
  static_assert(NQ * (KT + DP) <= 512, "TMEM columns");
};

struct PrefillItem {
  int req;         // < 0: no more items
  int kvh, piece, npieces;
  int tok0;        // first query token of the item inside its request
  int q_len, ctx;  // ctx: cached positions in front of the chunk (seq_len - q_len)
  int seq_len, q0; // q0: row of the request's first token
  int slot;        // workspace slot of the item's piece 0 (where there are several)
  int b, e0, e1;   // key tiles [b, e0) of row tile 0, [b, e1) of row tile 1
};

template <typename QT, int KV, int D>
__global__ void __launch_bounds__(kPrefillThreads, 1)
pa_prefill_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap vmap) {
  using SH = PrefillShape<D>;
  constexpr bool kFp8 = KV != kCache16;
  constexpr bool kE5 = KV == kCacheE5M2;
  constexpr bool kBf = !kFp8 && std::is_same_v<QT, __nv_bfloat16>;  // operand type: bf16, else f16
  constexpr bool kOutBf = std::is_same_v<QT, __nv_bfloat16>;
  constexpr int DP = SH::DP, NQ = SH::NQ, KT = SH::KT, NS = SH::kSlots;
  constexpr int kWs = 128 * (D * 2 + 8);  // workspace of one row tile's partial: O, then (m, l)
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ int cum[kPrefillMaxReqs + 1];  // 2 x (items before the request in place r), + 1 if it is cut into pieces
  __shared__ uint64_t s_bar[2 * NS + 19];
  __shared__ PrefillItem s_item[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_red[3][16];
  __shared__ int s_sort[kPrefillSortReqs];             // lengths, then items of the requests in their order
  __shared__ unsigned char s_order[kPrefillSortReqs];  // place -> request, where they are sorted

  const int tid = threadIdx.x, lane = tid & 31;
  // (through a shuffle, so that the compiler knows it is uniform in the warp)
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t bar0 = smem_u32(s_bar);
  auto kv_full = [&](uint32_t s) { return bar0 + 8u * s; };
  auto kv_empty = [&](uint32_t s) { return bar0 + 8u * (NS + s); };
  auto s_full = [&](int i) { return bar0 + 8u * (2 * NS + i); };
  auto p_full = [&](int i) { return bar0 + 8u * (2 * NS + 2 + i); };
  auto pv_done = [&](int i) { return bar0 + 8u * (2 * NS + 4 + i); };
  auto q_full = [&](int i) { return bar0 + 8u * (2 * NS + 6 + i); };
  auto item_full = [&](int i) { return bar0 + 8u * (2 * NS + 8 + i); };
  auto item_empty = [&](int i) { return bar0 + 8u * (2 * NS + 10 + i); };
  auto p_half = [&](int i) { return bar0 + 8u * (2 * NS + 12 + i); };
  const uint32_t tail_bar = bar0 + 8u * (2 * NS + 14);
  auto q_empty = [&](int i) { return bar0 + 8u * (2 * NS + 15 + i); };
  auto q_land = [&](int i) { return bar0 + 8u * (2 * NS + 17 + i); };
  constexpr bool kWiden = kFp8 && kOutBf;  // Q becomes f16, the operand type of an fp8 cache

  const uint32_t sq = smem_u32(smem);
  const uint32_t skv = sq + NQ * SH::kQBytes;
  if ((sq & 1023u) != 0) {  // (swizzles go by address bits)
    if (tid == 0) atomicExch(p.status, kStatusNoRing);
    return;
  }

  if (warp == 12) {
    if (lane == 0) {
      // (a warp arrives once, by its first lane: 128 arrivals on one barrier take a while)
      for (int s = 0; s < NS; ++s) {
        mbar_init(kv_full(s), 4);
        mbar_init(kv_empty(s), 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(s_full(i), 1);
        mbar_init(p_half(i), 4);
        mbar_init(p_full(i), 4);
        mbar_init(pv_done(i), 1);
        mbar_init(q_full(i), kWiden ? 2 : 1);
        mbar_init(q_land(i), 1);
        mbar_init(q_empty(i), 1);
        mbar_init(item_full(i), 1);
        mbar_init(item_empty(i), kWiden ? 15 : 14);
      }
      mbar_init(tail_bar, 1);
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(smem_u32(&s_tmem), 512);
  }
  if constexpr (DP != D) {
    // K's padding granule takes part in the product: zero, once (nobody writes it: K sits in the even
    // slots of the ring.  Q's comes as zeros, V's padding only gives columns that are dropped).
    static_assert(DP - D == 8 && NS % 2 == 0, "one padding granule; K and V in slots of their own");
    for (int i = tid; i < NS / 2 * KT; i += kPrefillThreads)
      *reinterpret_cast<uint4*>(smem + NQ * SH::kQBytes + (i / KT) * 2 * SH::kTileBytes + ((D / 8) * KT + i % KT) * 16) =
          make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  if (tid < 16) s_red[2][tid] = 0;  // (see the plan)
  __syncthreads();
  if (p.late_wait) grid_launch_dependents();
  else if (!p.early) grid_dependency();

  // ---- plan.  T tokens fill a row tile; a request has ceil(q_len / (NQ T)) row-tile groups per kv
  // head, and each of them npieces pieces.
  const int G = p.group, HK = p.num_kv_heads, S = p.num_reqs, B = p.block_size;
  const int b_shift = 31 - __clz(B);  // 16 or 32 tokens per block
  const int T = 128 / G, TT = NQ * T;
  static_assert(kPrefillThreads == kPrefillMaxReqs, "a thread to a request");
  int ql = 0, len = 0;
  if (tid < S) {
    ql = __ldcg(p.q_start + tid + 1) - __ldcg(p.q_start + tid);
    len = __ldcg(p.seq_lens + tid);
    if (tid < kPrefillSortReqs) s_sort[tid] = len;
  }
  const int n = (ql + TT - 1) / TT;  // groups
  int split_tiles;  // key tiles per piece (1 << 30: one piece per group)
  // Longest sequences first, where there are more groups than SMs: the last items of all are short ones
  // then, whatever the engine's order.  (60 decodes and three chunks of 150 to 700 tokens behind up to
  // 1500, 328 items: 124.5 -> 122 us; 6 fp8 chunks of 200 to 900 with a bias 147 -> 132; 12 bf16 chunks
  // 112 -> 108.5.  More than 64 requests keep their order, since each
  // thread would count over all of them.  Measured with a limit of 256: 128 equal prompts of 128 tokens 93.5 -> 95.3,
  // fp8 96.5 -> 102; requests of various lengths gain, 66 of 50 to 600 tokens behind up to 1500 0 to 4 %, 200 of 20
  // to 200 behind up to 3000 3 % (fp8 1 % more), 250 of 16 to 64 behind up to 2000 5 %, 100 of 2 to 20 behind up to
  // 6000 15 to 20 %, 309 -> 262: 64 is too low a line for those.)
  bool sorted = false;
  auto tiles_of = [&](int len) { return (max(len, 0) + KT - 1) / KT; };
  {
    // groups and key tiles of all requests: with fewer than four groups per SM the groups are cut
    // into pieces of an SM's share of the key tiles, but of no less than 768 keys: a piece costs a Q
    // load, a pipeline fill, a partial and its merge, about as much as 350 keys.
    // (Cuts of 512 keys and less: 128 tokens behind up to 1500 36 -> 33 us, but 550 tokens without context
    // 26 -> 32 and 1024 tokens behind 2048 at 2 kv heads 35 -> 50, where the pieces no longer run at once.
    // A search over the sizes with an estimate of the rounds costs every launch 1.4 us.)
    // Every piece of a group that is cut needs a slot of the workspace: s_red[2][k] counts the slots of
    // cuts of 768 keys x 1, 1.5, 2, 3, 4, 6 ..., and the finest from the share up that fits is taken.
    // (With a slot for every group, cut or not, nothing was cut beside 496 groups, or 31 on a small
    // region beside decodes: a 16-token chunk behind 32000 and 60 chunks of 32, 546 -> 169 us.)
    constexpr int kCut = 768 / KT;
    int groups = 0, work = 0;
    if (tid < S) {
      const int t = tiles_of(len);
      groups = n;
      work = n * ((t + tiles_of(len - ql + min(ql, TT)) + 1) / 2);
      const int q0 = (t + kCut - 1) / kCut, q1 = (t + kCut * 3 / 2 - 1) / (kCut * 3 / 2);
#pragma unroll 1
      for (int k = 0; k < 8 && t > kCut << k; ++k) {
        atomicAdd(&s_red[2][2 * k], n * HK * ((q0 + (1 << k) - 1) >> k));
        if (t > kCut * 3 / 2 << k) atomicAdd(&s_red[2][2 * k + 1], n * HK * ((q1 + (1 << k) - 1) >> k));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      groups += __shfl_xor_sync(0xffffffffu, groups, o);
      work += __shfl_xor_sync(0xffffffffu, work, o);
    }
    if (lane == 0) {
      s_red[0][warp] = groups;
      s_red[1][warp] = work;
    }
    __syncthreads();
    groups = work = 0;
    for (int w = 0; w < 16; ++w) {
      groups += s_red[0][w];
      work += s_red[1][w];
    }
    const int64_t all_work = int64_t(work) * HK, all_groups = int64_t(groups) * HK;
    sorted = S > 1 && S <= kPrefillSortReqs && all_groups > int64_t(gridDim.x);
    split_tiles = 1 << 30;
    if (all_groups < 4 * int64_t(gridDim.x)) {
      const int64_t up = all_work + gridDim.x - 1;
      const int want = up >> 32 == 0 ? int(uint32_t(up) / gridDim.x) : int(up / int64_t(gridDim.x));
      auto cut_of = [&](int k) { return ((k & 1) ? kCut * 3 / 2 : kCut) << (k >> 1); };
      const unsigned fit = __ballot_sync(
          0xffffffffu, lane < 16 && s_red[2][lane & 15] <= p.ws_slots && cut_of(lane + 1) > want);
      if (fit != 0) split_tiles = max(cut_of(__ffs(fit) - 1), want);
    }
    __syncthreads();  // (s_red is written again below)
  }
  auto pieces_of = [&](int len) -> unsigned {
    const unsigned t = tiles_of(len);
    return t <= unsigned(split_tiles) ? 1u : (t + split_tiles - 1u) / unsigned(split_tiles);
  };
  {
    const int pieces = pieces_of(len);
    int items = n * pieces * HK, cut = pieces > 1 ? 1 : 0;  // of the request in place tid
    if (sorted) {
      int place = 0;
      if (tid < S)
        for (int r = 0; r < S; ++r) place += s_sort[r] > len || (s_sort[r] == len && r < tid);
      __syncthreads();
      if (tid < S) {
        s_order[place] = tid;
        s_sort[place] = 2 * items + cut;
      }
      __syncthreads();
      items = tid < S ? s_sort[tid] >> 1 : 0;
      cut = tid < S ? s_sort[tid] & 1 : 0;
    }
    int incl = items;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_red[2][warp] = incl;
    __syncthreads();
    int run = incl - items;
    for (int w = 0; w < warp; ++w) run += s_red[2][w];
    if (tid < S) cum[tid] = 2 * run + cut;
    if (tid == kPrefillThreads - 1) cum[S] = 2 * (run + items);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int total = cum[S] >> 1;

  // item number -> what it covers.  Inside a request the row tiles run from the last to the first
  // (longest first), then the pieces, then the kv heads.
  auto decode = [&](int item) {
    PrefillItem it;
    auto starts = [&](int r) { return r < S && cum[r] >> 1 <= item; };  // (true up to the request of the item)
    int lo = 16 * (31 - __clz(__ballot_sync(0xffffffffu, starts(16 * lane))));
    lo += 31 - __clz(__ballot_sync(0xffffffffu, lane < 16 && starts(lo + lane)));
    it.req = sorted ? int(s_order[lo]) : lo;
    it.q0 = __ldcg(p.q_start + it.req);
    it.q_len = __ldcg(p.q_start + it.req + 1) - it.q0;
    it.seq_len = __ldcg(p.seq_lens + it.req);
    it.ctx = it.seq_len - it.q_len;
    const unsigned rel = item - (cum[lo] >> 1);
    unsigned gp = rel / unsigned(HK);
    it.kvh = rel - gp * HK;
    it.npieces = pieces_of(it.seq_len);
    it.piece = 0;
    if (it.npieces > 1) {
      const unsigned q = gp / unsigned(it.npieces);
      it.piece = gp - q * it.npieces;
      gp = q;
    }
    const int ngroups = (it.q_len + TT - 1) / TT;
    const int grp = ngroups - 1 - int(gp);
    // (the items of cut requests are counted only.  A table of the slots takes the static shared memory
    // past what a carve-out of 196 KiB holds at head size 128, and L1 shrinks to 28 KiB: 2 chunks of 64
    // behind 8192 take 98 us instead of 76.)
    it.slot = item - it.piece * HK;
    if (it.npieces > 1) {
      int others = 0;
      for (int r = lane; r < lo; r += 32)
        if ((cum[r] & 1) == 0) others += (cum[r + 1] >> 1) - (cum[r] >> 1);
      it.slot -= __reduce_add_sync(0xffffffffu, others);
    }
    it.tok0 = grp * TT;
    const int n = tiles_of(it.ctx + min(it.q_len, it.tok0 + TT));
    int e = n;
    it.b = 0;
    if (it.npieces > 1) {  // pieces of n / npieces tiles, the first ones of one more
      const int per = unsigned(n) / unsigned(it.npieces), more = n - per * it.npieces;
      it.b = it.piece * per + min(it.piece, more);
      e = it.b + per + (it.piece < more ? 1 : 0);
    }
    auto end_of = [&](int i) {
      const int t0 = it.tok0 + i * T;
      return i < NQ && t0 < it.q_len ? max(it.b, min(e, tiles_of(it.ctx + min(it.q_len, t0 + T)))) : it.b;
    };
    it.e0 = end_of(0);
    it.e1 = end_of(1);
    return it;
  };
  bool ok = true;
  // All roles wait as whole warps and leave as whole warps (TMEM accesses are warp-collective).
  auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
    const bool got = __all_sync(0xffffffffu, mbar_spin(bar, parity));
    if (!got) {
      ok = false;
      if (lane == 0) atomicExch(p.status, kStatusMbarTimeout);
    }
    return got;
  };
  auto arrive = [&](uint32_t bar) {  // once per warp, for everything its lanes have done
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  // Items of this CTA: warp 13 draws them, works out what they cover and puts that into a ring of two;
  // the other roles look there and give the place back when they are through with an item.
  int n_item = 0;  // items received so far
  auto have_item = [&]() -> bool {
    return wait(item_full(n_item & 1), (n_item >> 1) & 1) && s_item[n_item & 1].req >= 0;
  };
  auto item_done = [&]() {
    arrive(item_empty(n_item & 1));
    ++n_item;
  };

  if (warp < 8) {
    // ================================================= softmax: one thread per row of tile wg
    reg_inc<PrefillRegs<kFp8>::kSoftmax>();
    const int wg = warp >> 2;
    const int row = tid & 127;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem + lane_off + uint32_t(wg * KT);
    const uint32_t t_o = tmem + lane_off + uint32_t(NQ * KT + wg * DP);
    const float c = p.scale * kLog2e * (kFp8 ? __ldcg(p.k_scale) : 1.f);
    const bool biased = p.alibi != nullptr || !(c > 0.f);  // the maximum is taken of the scaled values then
    const float v_scale = kFp8 ? __ldcg(p.v_scale) : 1.f;
    const bool row_used = wg < NQ && row < T * G;
    const int row_tok = row / G, row_head = row % G;
    uint32_t n_s = 0, n_pv = 0;  // S tiles received, PV products issued for this row tile

    while (ok && have_item()) {
      const PrefillItem& it = s_item[n_item & 1];
      const int b = it.b, e = wg == 0 ? it.e0 : it.e1;
      const int tok = it.tok0 + wg * T + row_tok;
      const bool valid = row_used && tok < it.q_len;
      const int pos = valid ? it.ctx + tok : -1;                     // last key of this row
      const int pos_first = it.ctx + it.tok0 + wg * T;               // ... of the tile's first row
      const int head = it.kvh * G + row_head;
      const float slope = (p.alibi != nullptr && valid) ? __ldcg(p.alibi + head) * kLog2e : 0.f;
      float m = -INFINITY, l = 0.f;
      bool unset = true;  // a row of this warp has no maximum yet: every logit so far was masked or -inf
      for (int j = b; j < e; ++j) {
        if (!wait(s_full(wg), n_s & 1)) break;
        ++n_s;
        tc_fence_after();
        // The whole row of S goes to registers at once.  After the first tile the running maximum mostly
        // stands: for 16-bit caches without a bias the exponentials of the first half start with it as it
        // is; their sum and, beside them, the maximum of the second half tell whether it was too low (by
        // 2^12: P and its sums hold larger values as exactly).  Then, and as long as a row has no maximum at
        // all (the first tile, and those behind it while logits are -inf), the maximum of the row is taken
        // first.
        // (8192-token step 363 -> 353 us, with no gain for fp8 caches; with a bias the maximum grows with
        // every tile, 148 -> 177.  Exponentials by a polynomial on the FMA pipe instead of the special
        // function unit, a quarter of them: 354 -> 368; the kernel runs into the power limit, and without
        // any exponentials it would take 336.)
        constexpr int NC = KT / 32;
        const int key0 = j * KT;
        float x[NC][32], cc = c, nm = 0.f;
        float2 sa, sb;
        uint32_t w[NC][16];
        auto exps = [&](int ch, int k) {
          const float2 t = ffma2(make_float2(x[ch][k], x[ch][k + 1]), make_float2(cc, cc), make_float2(nm, nm));
          const float2 e2 = make_float2(fast_exp2(t.x), fast_exp2(t.y));
          if (k & 2) sb = fadd2(sb, e2); else sa = fadd2(sa, e2);
          w[ch][k / 2] = pack2<kBf>(e2.x, e2.y);
        };
        for (bool look = kFp8 || biased || unset;; look = true) {
#pragma unroll
          for (int ch = 0; ch < NC; ++ch) tmem_ld32(t_s + ch * 32, x[ch]);
          int last = pos - key0;  // last column of this row that counts
          cc = c;                 // (goes through the wait for the TMEM loads, see tmem_landed)
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          tmem_landed(m4, cc, last);
          if (biased) {  // t = x c + slope (key - pos)
            const float base = slope * -float(last);
#pragma unroll
            for (int ch = 0; ch < NC; ++ch)
#pragma unroll
              for (int k = 0; k < 32; ++k) x[ch][k] = fmaf(slope, float(ch * 32 + k), fmaf(x[ch][k], cc, base));
            cc = 1.f;
          }
          if (key0 + KT - 1 > pos_first) {  // only the tiles at the causal edge of a row tile need a mask
            asm volatile("");               // (a branch in fact, not 128 selects for every tile)
#pragma unroll
            for (int ch = 0; ch < NC; ++ch)
#pragma unroll
              for (int k = 0; k < 32; ++k) x[ch][k] = ch * 32 + k <= last ? x[ch][k] : -INFINITY;
          }
          if (kFp8 || look) {
            asm volatile("");
            float h4[4] = {m4[0], m4[1], m4[2], m4[3]};
#pragma unroll
            for (int ch = 0; ch < NC; ++ch)
#pragma unroll
              for (int k = 0; k < 32; k += 2) h4[k / 2 & 3] = fmax3(h4[k / 2 & 3], x[ch][k], x[ch][k + 1]);
            const float mx = fmax3(fmaxf(h4[0], h4[1]), h4[2], h4[3]) * cc;
            // raise the maximum, and rescale what has been summed
            const bool grow = mx > m + (kFp8 || biased ? 8.f : 0.f) || (m == -INFINITY && mx > m);
            if (__any_sync(0xffffffffu, grow)) {
              const float m_new = fmaxf(m, mx);
              const float alpha = m_new == -INFINITY ? 1.f : fast_exp2(m - m_new);
              m = m_new;
              l *= alpha;
              if (j > b) {
                if (!wait(pv_done(wg), (n_pv - 1) & 1)) break;
                tc_fence_after();
#pragma unroll 1
                for (int ch = 0; ch < DP / 16; ++ch) {
                  float o[16];
                  tmem_ld16(t_o + ch * 16, o);
#pragma unroll
                  for (int k = 0; k < 16; ++k) o[k] *= alpha;
                  tmem_st16(t_o + ch * 16, o);
                }
                tmem_wait_st();
              }
            }
            if (!kFp8) unset = __any_sync(0xffffffffu, valid && m == -INFINITY);
          }
          nm = m == -INFINITY ? 0.f : -m;
          sa = sb = make_float2(0.f, 0.f);
#pragma unroll
          for (int ch = 0; ch < NC / 2; ++ch)
#pragma unroll
            for (int k = 0; k < 32; k += 2) {
              exps(ch, k);
              if (!kFp8) m4[k / 2 & 3] = fmax3(m4[k / 2 & 3], x[NC / 2 + ch][k], x[NC / 2 + ch][k + 1]);
            }
          const float mx = fmax3(fmaxf(m4[0], m4[1]), m4[2], m4[3]) * cc;
          const bool low = (sa.x + sa.y) + (sb.x + sb.y) > 4096.f || mx > m + 12.f;
          if (kFp8 || look || !__any_sync(0xffffffffu, low)) break;
        }
        if (!ok) break;
        // (P's columns lie over S columns: 16 a chunk of 32)
#pragma unroll
        for (int ch = 0; ch < NC; ++ch) {
          if (ch >= NC / 2) {
#pragma unroll
            for (int k = 0; k < 32; k += 2) exps(ch, k);
          }
          tmem_st16(t_s + ch * 16, w[ch]);
          if (ch == NC / 2 - 1 || ch == NC - 1) {
            tmem_wait_st();
            tc_fence_before();
            arrive(ch == NC - 1 ? p_full(wg) : p_half(wg));
          }
        }
        l += (sa.x + sa.y) + (sb.x + sb.y);
        ++n_pv;
      }
      if (!ok) break;
      if (wg >= NQ) {
        item_done();
        continue;
      }
      // ---- results
      const bool any = e > b;
      if (any) {
        if (!wait(pv_done(wg), (n_pv - 1) & 1)) break;
        tc_fence_after();
      }
      const bool whole = it.npieces == 1;
      const float inv = v_scale * __fdividef(1.f, l + 1e-6f);
      const int64_t out_row = (int64_t(it.q0 + tok) * p.num_heads + head) * D;
      const int slot = it.slot;
      unsigned char* part = p.ws + (size_t(slot + it.piece * HK) * NQ + wg) * kWs;
      QT* dst = static_cast<QT*>(p.out) + out_row;
      // A partial lies as [16 bytes of the head][row] for the 32 rows of a warp, so that a warp's stores,
      // and its loads when it merges, are whole lines.  (Rows one after the other: 32 lines an
      // instruction; 64 tokens behind 8192, 9 pieces, 71 us instead of 47.)
      constexpr int kWarpPart = 32 * D * 2;
      const int mine = (warp & 3) * kWarpPart + lane * 16;
      // 32 bytes a store where rows allow it: a row is another 128-byte line for each lane, whatever it
      // stores there
      const bool wide = D % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
      if (any || whole) {
        constexpr int NCO = DP / 16, CH = NCO % 4 == 0 ? 4 : (NCO % 3 == 0 ? 3 : NCO);  // chunks read at a time
        static_assert(CH <= 7, "registers");
#pragma unroll 1
        for (int c0 = 0; c0 < NCO; c0 += CH) {
          float o[CH][16], keep[4] = {inv, 0.f, 0.f, 0.f};
          float inv2 = inv;
          int dummy = 0;
          if (any) {
#pragma unroll
            for (int k = 0; k < CH; ++k) tmem_ld16_start(t_o + (c0 + k) * 16, o[k]);
            tmem_landed(keep, inv2, dummy);
          } else {
#pragma unroll
            for (int k = 0; k < CH; ++k)
#pragma unroll
              for (int i = 0; i < 16; ++i) o[k][i] = 0.f;
          }
          if (valid) {
#pragma unroll
            for (int k = 0; k < CH; ++k) {
              uint32_t w[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) w[i] = pack2<kOutBf>(o[k][2 * i] * inv2, o[k][2 * i + 1] * inv2);
              QT* d = dst + (c0 + k) * 16;
              if (!whole) {
                uint4* pd = reinterpret_cast<uint4*>(part + mine + (c0 + k) * 2 * 512);
                pd[0] = make_uint4(w[0], w[1], w[2], w[3]);
                if (D % 16 == 0 || (c0 + k) * 16 + 8 < D) pd[32] = make_uint4(w[4], w[5], w[6], w[7]);
              } else if (wide) {
                st_global32(d, w);
              } else {
                reinterpret_cast<uint4*>(d)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                if (D % 16 == 0 || (c0 + k) * 16 + 8 < D) reinterpret_cast<uint4*>(d)[1] = make_uint4(w[4], w[5], w[6], w[7]);
              }
            }
          }
        }
        tc_fence_before();  // (ordered before the next item's p_half, which frees O)
      }
      if (!whole) {
        float* stats = reinterpret_cast<float*>(part + 128 * D * 2);
        if (valid) reinterpret_cast<float2*>(stats)[row] = make_float2(m, any ? l : 0.f);
        // the rows of a warp are merged by the warp that delivers their last piece
        __syncwarp();
        unsigned old = 0;
        unsigned* cnt = p.arrive + (size_t(slot) * NQ + wg) * 4 + (warp & 3);
        if (lane == 0) {
          __threadfence();  // (for the whole warp: __syncwarp orders its stores before it)
          old = atomicAdd(cnt, 1u);
          if (old == unsigned(it.npieces - 1)) *cnt = 0;  // re-arm for the next launch
          __threadfence();
        }
        __syncwarp();  // the other lanes' loads of partials come after lane 0's fence (a shuffle orders no memory)
        old = __shfl_sync(0xffffffffu, old, 0);
        if (old == unsigned(it.npieces - 1) && valid) {
          const unsigned char* base = p.ws + (size_t(slot) * NQ + wg) * kWs;
          const size_t step = size_t(HK) * NQ * kWs;
          // statistics of eight pieces at a time (independent loads), online
          float mx = -INFINITY, total_l = 0.f;
#pragma unroll 1
          for (int k0 = 0; k0 < it.npieces; k0 += 8) {
            float2 ml[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
              ml[k] = __ldcg(reinterpret_cast<const float2*>(base + min(k0 + k, it.npieces - 1) * step + 128 * D * 2) + row);
            float m_new = mx;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (k0 + k < it.npieces && ml[k].y > 0.f) m_new = fmaxf(m_new, ml[k].x);
            if (m_new == -INFINITY) continue;
            total_l *= fast_exp2(mx - m_new);
            mx = m_new;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (k0 + k < it.npieces && ml[k].y > 0.f) total_l += ml[k].y * fast_exp2(ml[k].x - mx);
          }
          const float winv = __fdividef(1.f, total_l + 1e-6f);
          // up to 64 bytes of the row and six pieces at a time: 24 independent loads on their way
          constexpr int NCH = D / 8, MC = NCH % 4 == 0 ? 4 : (NCH % 2 == 0 ? 2 : 3), MP = 6;
          static_assert(NCH % MC == 0, "no rest");
#pragma unroll 1
          for (int c0 = 0; c0 < NCH; c0 += MC) {
            float acc[MC][8];
#pragma unroll
            for (int c = 0; c < MC; ++c)
#pragma unroll
              for (int z = 0; z < 8; ++z) acc[c][z] = 0.f;
#pragma unroll 1
            for (int k0 = 0; k0 < it.npieces; k0 += MP) {
              uint4 x[MP][MC];
              float w[MP];
#pragma unroll
              for (int k = 0; k < MP; ++k) {
                const unsigned char* pk = base + min(k0 + k, it.npieces - 1) * step;
                const float2 ml = __ldcg(reinterpret_cast<const float2*>(pk + 128 * D * 2) + row);
#pragma unroll
                for (int c = 0; c < MC; ++c)
                  x[k][c] = __ldcg(reinterpret_cast<const uint4*>(pk + mine + (c0 + c) * 512));
                // (a piece in which this row has no key has written no output)
                w[k] = k0 + k < it.npieces && ml.y > 0.f ? ml.y * fast_exp2(ml.x - mx) * winv : 0.f;
              }
#pragma unroll
              for (int k = 0; k < MP; ++k) {
                if (w[k] == 0.f) continue;
#pragma unroll
                for (int c = 0; c < MC; ++c) {
                  const QT* xe = reinterpret_cast<const QT*>(&x[k][c]);
#pragma unroll
                  for (int z = 0; z < 8; ++z) acc[c][z] += w[k] * to_f32(xe[z]);
                }
              }
            }
#pragma unroll
            for (int c = 0; c < MC; ++c)
              *reinterpret_cast<uint4*>(dst + (c0 + c) * 8) =
                  make_uint4(pack2<kOutBf>(acc[c][0], acc[c][1]), pack2<kOutBf>(acc[c][2], acc[c][3]),
                             pack2<kOutBf>(acc[c][4], acc[c][5]), pack2<kOutBf>(acc[c][6], acc[c][7]));
          }
        }
        __syncwarp();
      }
      item_done();
    }
  } else if (warp < 12) {
    // ================================================= producers: K and V tiles into shared memory
    reg_dec<PrefillRegs<kFp8>::kProducer>();
    const int pt = tid - 256;  // 0 .. 127
    uint32_t n_half = 0;       // halves (K or V tiles) put on their way
    uint32_t n_tail = 0;       // last tiles of a sequence that ended inside a page
    const char* kb = static_cast<const char*>(p.kc);
    const char* vb = static_cast<const char*>(p.vc);
    constexpr int ES = kFp8 ? 1 : 2;
    // K tiles of 16-bit caches are announced when their copies have landed, up to two later; before
    // the warp waits for anything, all of them are (the MMAs may be waiting for just those).
    uint32_t n_k = 0, n_told = 0;  // K tiles put on their way, announced
    auto announce = [&]() {
      fence_proxy_async();
      arrive(kv_full(2 * n_told % NS));
      ++n_told;
    };
    auto announce_all = [&]() {
      if (n_k - n_told >= 2) {
        cp_async_wait<1>();
        while (n_k - n_told > 1) announce();
      }
      if (n_k != n_told) {
        cp_async_wait<0>();
        announce();
      }
    };
    auto wait_slot = [&](uint32_t h) -> bool {
      const uint32_t use = h / NS;  // times the slot has been filled before
      if (use == 0) return true;
      if constexpr (!kFp8) {
        if (!__all_sync(0xffffffffu, mbar_test(kv_empty(h % NS), (use - 1) & 1))) announce_all();
      }
      return wait(kv_empty(h % NS), (use - 1) & 1);
    };
    auto slot_of = [&](uint32_t h) { return skv + (h % NS) * SH::kTileBytes; };
    if (!kFp8 && warp == 8) fence_proxy_async_global();  // (V, under late_wait)
    while (ok && have_item()) {
      const PrefillItem it = s_item[n_item & 1];
      const int* bt = p.block_tables + int64_t(it.req) * p.max_blocks_per_seq;
      const int64_t head_off = int64_t(it.kvh) * p.kv_head_stride * ES;
      const int e = max(it.e0, it.e1);
      auto block_of = [&](int key) { return key < it.seq_len ? __ldcg(bt + (key >> b_shift)) : 0; };
      auto page = [&](const char* base, int blk) {
        return base + int64_t(blk) * p.kv_block_stride * ES + head_off;
      };
      if constexpr (!kFp8) {
        // K: a thread owns one key and walks along its 16-byte granules (128 bytes of shared memory per
        // 8 threads).  V: pages of 16 keys, each one copy by tensor map, whose rows of 16 keys are a K
        // step of the product (32-byte swizzle); issued by the first warp.  (V by 16-byte cp.async came
        // in half sectors and kept the load/store unit from the softmax: 8192-token step 444 -> 392 us.  K
        // by bulk copies of 256 bytes, the run of a granule in a page, takes 835: 128 of them a tile.)
        constexpr int NP = KT / 16;  // pages per tile
        const int kt = pt % KT, kg = pt / KT;
        int k_blk = block_of(it.b * KT + kt), v_blk = block_of(it.b * KT + lane % NP * 16);
        if (p.early) grid_dependency();  // (from here on K and V; returns at once when it has done so before)
        for (int j = it.b; j < e && ok; ++j) {
          {
            const int key = j * KT + kt;
            const char* src = page(kb, k_blk) + (kg * B + (key & (B - 1))) * 16;
            const int bytes = key < it.seq_len ? 16 : 0;
            if (j + 1 < e) k_blk = block_of(key + KT);
            if (!wait_slot(n_half)) break;
            uint32_t dst = slot_of(n_half) + (kg * KT + kt) * 16;
#pragma unroll 4
            for (int g = kg; g < D / 8; g += 128 / KT) {
              cp_async16(dst, src, bytes);
              dst += 128 * 16;
              src += (128 / KT) * B * 16;
            }
            cp_async_commit();
            ++n_half;
            ++n_k;
            if (n_k - n_told > 1) {
              cp_async_wait<1>();
              announce();
            }
          }
          const int key = j * KT + lane % NP * 16;
          const int cur = v_blk;
          if (j + 1 < e) v_blk = block_of(key + KT);
          if (!wait_slot(n_half)) break;
          {
            // only pages with a key of the sequence are copied
            const int pages = min(NP, (it.seq_len - j * KT + 15) / 16);
            const int left = it.seq_len - j * KT - (pages - 1) * 16;  // keys of the last page that exist
            const bool cut = left < 16;
            const uint32_t full = kv_full(n_half % NS), bar = cut ? tail_bar : full;
            if (warp != 8) {
              arrive(full);
              ++n_half;
              continue;
            }
            if (lane == 0) mbar_expect_tx(bar, pages * D * 32);
            __syncwarp();
            if (lane < pages) tma_load4(slot_of(n_half) + lane * DP * 32, &vmap, key & (B - 1), 0, it.kvh, cur, bar);
            __syncwarp();
            if (cut) {
              // keys past the end become zeros (stale bytes could be NaN)
              announce_all();
              if (!wait(bar, n_tail++ & 1)) break;
              const uint32_t last = slot_of(n_half) + (pages - 1) * DP * 32;
              for (int d = lane; d < D; d += 32) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const uint32_t at = last + d * 32 + (h ^ (d >> 2 & 1)) * 16;
                  const int n = left - 8 * h;  // keys of this half row that exist
                  uint4 x = ld_shared16(at);
                  x.x = n >= 2 ? x.x : (n == 1 ? x.x & 0xffffu : 0u);
                  x.y = n >= 4 ? x.y : (n == 3 ? x.y & 0xffffu : 0u);
                  x.z = n >= 6 ? x.z : (n == 5 ? x.z & 0xffffu : 0u);
                  x.w = n >= 8 ? x.w : (n == 7 ? x.w & 0xffffu : 0u);
                  st_shared16(at, x);
                }
              }
              fence_proxy_async();
              arrive(full);
            }
            ++n_half;
          }
        }
      } else {
        // fp8: 16-byte loads into registers (the next half is always in flight), widened to two
        // 16-byte granules of f16.  K: a thread owns one key; V: 16 keys and every 16th dimension.
        const int kt = pt % KT, kg = pt / KT;
        constexpr int KN = (D / 16 + 128 / KT - 1) / (128 / KT);
        constexpr int VJ = KT / 16;
        constexpr int VDS = 128 / VJ;           // threads that share a 16-key group
        const int vj = pt / VDS, vd = pt % VDS;
        constexpr int VN = (D + VDS - 1) / VDS;
        uint4 kr[KN], vr[VN];
        auto get_k = [&](int j) {
          const int key = j * KT + kt;
          const char* src = page(kb, block_of(key)) + (key & (B - 1)) * 16;
#pragma unroll
          for (int i = 0; i < KN; ++i) {
            const int g = kg + i * (128 / KT);
            if (key < it.seq_len && g < D / 16) kr[i] = __ldcg(reinterpret_cast<const uint4*>(src + int64_t(g) * B * 16));
            else kr[i] = make_uint4(0, 0, 0, 0);
          }
        };
        auto get_v = [&](int j) {
          const int key = j * KT + vj * 16;
          const char* src = page(vb, block_of(key)) + (key & (B - 1));
#pragma unroll
          for (int i = 0; i < VN; ++i) {
            const int d = vd + i * VDS;
            if (key < it.seq_len && d < D) vr[i] = __ldcg(reinterpret_cast<const uint4*>(src + int64_t(d) * B));
            else vr[i] = make_uint4(0, 0, 0, 0);
          }
        };
        auto widen = [&](const uint4& x, uint4& lo, uint4& hi) {
          fp8x4_to_f16<kE5>(x.x, lo.x, lo.y);
          fp8x4_to_f16<kE5>(x.y, lo.z, lo.w);
          fp8x4_to_f16<kE5>(x.z, hi.x, hi.y);
          fp8x4_to_f16<kE5>(x.w, hi.z, hi.w);
        };
        if (p.early) grid_dependency();
        if (it.b < e) {
          get_k(it.b);
          get_v(it.b);
        }
        for (int j = it.b; j < e && ok; ++j) {
          if (!wait_slot(n_half)) break;
          {
            const uint32_t dst = slot_of(n_half) + kt * 16;
#pragma unroll
            for (int i = 0; i < KN; ++i) {
              const int g = kg + i * (128 / KT);
              if (D / 16 % (128 / KT) == 0 || g < D / 16) {
                uint4 lo, hi;
                widen(kr[i], lo, hi);
                st_shared16(dst + (2 * g) * KT * 16, lo);
                st_shared16(dst + (2 * g + 1) * KT * 16, hi);
              }
            }
            fence_proxy_async();
            arrive(kv_full(n_half % NS));
            ++n_half;
            if (j + 1 < e) get_k(j + 1);
          }
          if (!wait_slot(n_half)) break;
          {
            const uint32_t dst = slot_of(n_half) + 2 * vj * DP * 16;
            const int left = it.seq_len - (j * KT + vj * 16);  // keys of the group that exist
#pragma unroll
            for (int i = 0; i < VN; ++i) {
              const int d = vd + i * VDS;
              if (D % VDS == 0 || d < D) {
                uint4 x = vr[i];
                if (left < 16) {  // keys past the end: zeros
                  auto keep = [&](uint32_t w, int at) {
                    const int n = left - at;
                    return n >= 4 ? w : (n <= 0 ? 0u : w & (0xffffffffu >> (32 - 8 * n)));
                  };
                  x = make_uint4(keep(x.x, 0), keep(x.y, 4), keep(x.z, 8), keep(x.w, 12));
                }
                uint4 lo, hi;
                widen(x, lo, hi);
                st_shared16(dst + d * 16, lo);
                st_shared16(dst + (DP + d) * 16, hi);
              }
            }
            fence_proxy_async();
            arrive(kv_full(n_half % NS));
            ++n_half;
            if (j + 1 < e) get_v(j + 1);
          }
        }
      }
      if (!ok) break;
      if constexpr (!kFp8) announce_all();  // (the next item may be drawn only when they have arrived)
      item_done();
    }
    if constexpr (!kFp8) {  // nobody leaves with copies on their way (after a wait that ran out, too)
      cp_async_wait_all();
      if (warp == 8)
        for (uint32_t h = n_half < NS ? 0 : n_half - NS; h < n_half; ++h) mbar_spin(kv_full(h % NS), (h / NS) & 1);
    }
  } else {
    reg_dec<PrefillRegs<kFp8>::kMma>();
    if (warp == 12) {
    // ================================================= the MMA warp.  All lanes run along, so that
    // operand descriptors stay in uniform registers, and one elected lane issues: with a single
    // lane running, moving them there cost 95 cycles an MMA of 64.  Uniform registers belong to the
    // warp: after every block of the elected lane the warp converges before anything else runs.
    const uint32_t idesc_s = mma_idesc(kBf, 128, KT);
    const uint32_t idesc_o = mma_idesc(kBf, 128, DP);
    uint32_t n_h = 0, n_q0 = 0, n_q1 = 0, n_p0 = 0, n_p1 = 0;  // halves, Q tiles, P tiles
    auto uniform = [](uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); };
    auto commit = [&](uint32_t bar) {
      if (elect_one()) mma_commit(bar);
      __syncwarp();
    };
    const uint64_t q_desc = SH::kQBox == 64 ? smem_desc_sw128(sq) : smem_desc_sw32(sq, 256);
    auto q_step = [](int ks) {  // where K step ks lies, in 16-byte units
      return SH::kQBox == 64 ? ks / 4 * (128 * 128 / 16) + ks % 4 * 2 : ks * (128 * 32 / 16);
    };
    const uint64_t k_desc = smem_desc(skv, KT * 16, 128);
    const uint64_t v_desc = kFp8 ? smem_desc(skv, DP * 16, 128) : smem_desc_sw32(skv, 256);
    auto wait_half = [&](uint32_t h) { return wait(kv_full(h % NS), (h / NS) & 1); };
    auto qk = [&](int i, uint32_t h) {
      const uint64_t kd = k_desc + uniform((h % NS) * (SH::kTileBytes >> 4));
      const uint64_t qd = q_desc + i * (SH::kQBytes >> 4);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < DP / 16; ++ks)
          mma_ss(tmem + i * KT, qd + q_step(ks), kd + ks * 2 * KT, idesc_s, ks > 0);
        mma_commit(s_full(i));
      }
      __syncwarp();
    };
    // half of the keys of a tile: the first while the softmax works on the second (`steps`: pages of 16
    // keys that the tile has)
    auto pv = [&](int i, uint32_t h, int half, int steps, bool more) {
      const uint64_t vd = v_desc + uniform((h % NS) * (SH::kTileBytes >> 4));
      if (elect_one()) {
        constexpr int NK = KT / 32;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const int ks = half * NK + k;
          if (kFp8 || ks < steps)
            mma_ts(tmem + NQ * KT + i * DP, tmem + i * KT + ks * 8, vd + ks * 2 * DP, idesc_o, more || ks > 0);
        }
        if (half == 1) mma_commit(pv_done(i));
      }
      __syncwarp();
    };
    while (ok && have_item()) {
      struct { int b, e0, e1, seq_len; } it;
      {
        const PrefillItem& from = s_item[n_item & 1];
        it.b = uniform(from.b);
        it.e0 = uniform(from.e0);
        it.e1 = uniform(from.e1);
        it.seq_len = uniform(from.seq_len);
      }
      const int e = max(it.e0, it.e1);
      if (it.b < e) {
        if (!wait_half(n_h)) break;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const int ei = i == 0 ? it.e0 : it.e1;
          if (it.b >= ei) continue;
          if (!wait(q_full(i), (i == 0 ? n_q0++ : n_q1++) & 1)) break;
          tc_fence_after();
          qk(i, n_h);
          if (it.b + 1 == ei) commit(q_empty(i));
        }
        if (!ok) break;
        commit(kv_empty(n_h % NS));
        ++n_h;
      }
      for (int j = it.b; j < e; ++j) {
        // V tile j is half n_h, K tile j + 1 half n_h + 1
        if (!wait_half(n_h)) break;
        bool have_k = false;
        const int steps = (it.seq_len - j * KT + 15) / 16;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const int ei = i == 0 ? it.e0 : it.e1;
          uint32_t& n_p = i == 0 ? n_p0 : n_p1;
          if (!ok || j >= ei) continue;
          if (!wait(p_half(i), n_p & 1)) continue;
          tc_fence_after();
          pv(i, n_h, 0, steps, j > it.b);
          if (!wait(p_full(i), n_p & 1)) continue;
          ++n_p;
          tc_fence_after();
          pv(i, n_h, 1, steps, true);
          if (j + 1 < ei) {
            if (!have_k && !wait_half(n_h + 1)) continue;
            have_k = true;
            qk(i, n_h + 1);
            if (j + 2 == ei) commit(q_empty(i));
          }
        }
        if (!ok) break;
        commit(kv_empty(n_h % NS));
        ++n_h;
        if (have_k) {
          commit(kv_empty(n_h % NS));
          ++n_h;
        }
      }
      if (!ok) break;
      item_done();
    }
    } else if (warp == 13) {
    // ================================================= draws items and works out what they cover
    // (when everybody is through with the item before the one in work: any earlier, and the SMs end
    // less evenly)
    int item = blockIdx.x < unsigned(total) ? int(blockIdx.x) : INT32_MAX;
    for (;; ++n_item) {
      const int slot = n_item & 1;
      if (n_item >= 2 && !wait(item_empty(slot), ((n_item >> 1) - 1) & 1)) break;
      if (n_item >= 1) {
        unsigned ticket = 0;
        if (lane == 0) ticket = atomicAdd(p.sched, 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        item = int(min(ticket + gridDim.x, unsigned(INT32_MAX)));
      }
      PrefillItem it{};
      it.req = -1;
      if (item < total) it = decode(item);
      if (lane == 0) {
        s_item[slot] = it;
        mbar_arrive(item_full(slot));
      }
      __syncwarp();
      if (item >= total) break;
    }
    } else {
    // ================================================= Q into shared memory (warp 14), as soon as the
    // last product with the Q before it is through: a tile's tokens and heads are a box of a tensor
    // map.  (16-byte cp.async by two warps: 1600 cycles to issue, 3000 until they landed; by the softmax
    // warpgroups after their last tile 6500, which nothing hid.)  bf16 becomes f16 in place for an
    // fp8 cache, half a tile by each of warps 14 and 15.
    uint32_t n_q[2] = {0, 0};
    fence_proxy_async_global();  // (Q, under late_wait and early)
    while (ok && (kWiden || warp == 14) && have_item()) {
      const PrefillItem& it = s_item[n_item & 1];
      const bool has[2] = {it.e0 > it.b, it.e1 > it.b};
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        if (!has[i]) continue;
        const uint32_t land = kWiden ? q_land(i) : q_full(i);
        if (warp == 14) {
          if (n_q[i] > 0 && !wait(q_empty(i), (n_q[i] - 1) & 1)) break;
          constexpr int NB = DP / SH::kQBox;
          if (lane == 0) {
            mbar_expect_tx(land, NB * SH::kQBox * 2 * T * G);
#pragma unroll
            for (int x = 0; x < NB; ++x)
              tma_load3(sq + i * SH::kQBytes + x * 128 * SH::kQBox * 2, &qmap, x * SH::kQBox, it.kvh * G,
                        it.q0 + it.tok0 + i * T, land);
          }
          __syncwarp();
        }
        if constexpr (kWiden) {
          if (!wait(land, n_q[i] & 1)) break;
          const uint32_t at = sq + i * SH::kQBytes + (warp - 14) * (SH::kQBytes / 2) + lane * 16;
#pragma unroll 4
          for (int o = 0; o < SH::kQBytes / 2; o += 512) {
            const uint4 v = ld_shared16(at + o);
            auto f16 = [](uint32_t w) { return pack2<false>(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); };
            st_shared16(at + o, make_uint4(f16(v.x), f16(v.y), f16(v.z), f16(v.w)));
          }
          fence_proxy_async();
          arrive(q_full(i));
        }
        ++n_q[i];
      }
      if (!ok) break;
      item_done();
    }
    if (warp == 14) {  // nobody leaves with copies on their way
#pragma unroll
      for (int i = 0; i < NQ; ++i)
        if (n_q[i] > 0) mbar_spin(kWiden ? q_land(i) : q_full(i), (n_q[i] - 1) & 1);
    }
    }
  }

  if (p.late_wait || p.early) grid_dependency_wait();
  // ---- everything issued has been waited for by the softmax warpgroups (or a wait ran out)
  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (tid == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(p.sched + 1, 1u);
    if (prev == gridDim.x - 1) {
      p.sched[0] = 0;
      p.sched[1] = 0;
      __threadfence();
    }
  }
}

}  // namespace b200pa
