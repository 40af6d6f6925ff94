// Host entry of attention over a step whose requests bring several query tokens each: the requests
// in front that bring one go to the decode kernel, the others to the prefill kernel.
#include <algorithm>
#include <cstdint>

#include "launch_state.cuh"
#include "prefill_inst.cuh"
#include "tensor_map.cuh"

namespace b200pa {

cudaError_t prefill_v_map(const PrefillParams& p, int head_size, CUtensorMap* map) {
  return tensor_map<4>(map, p.vc, {p.block_size, head_size, p.num_kv_heads, INT32_MAX},
                       {p.block_size, p.kv_head_stride, p.kv_block_stride}, {16, head_size, 1, 1}, CU_TENSOR_MAP_SWIZZLE_32B);
}

cudaError_t prefill_q_map(const PrefillParams& p, int head_size, int box, CUtensorMap* map) {
  return tensor_map<3>(map, p.q, {head_size, p.num_heads, p.num_tokens}, {head_size, p.q_stride},
                       {box, p.group, 128 / p.group}, box == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// A dimension of size 1 may come with any stride, 0 among them; a tensor map wants one that it can hold.
// (num_tokens 0: not known)
static b200pa_attn_args with_plain_strides(b200pa_attn_args a, int num_tokens) {
  if (a.num_kv_heads == 1) a.kv_head_stride = int64_t(a.head_size) * a.block_size;
  if (num_tokens == 1) a.q_stride = int64_t(a.num_heads) * a.head_size;
  return a;
}

// The prefill kernel for a call's shape and alignments, or none.  16-byte accesses: pages, rows of Q and
// of the output; cache offsets inside a block are shifts.  The strides of Q and of a 16-bit cache have to
// fit a tensor map (positive, below 2^40 bytes).
static PrefillKernelInfo find_prefill(const b200pa_attn_args& a) {
  const int es = a.kv_dtype == B200PA_KV_AUTO ? 2 : 1;
  auto al = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; };
  const bool fits = (a.block_size == 16 || a.block_size == 32) && a.num_heads / a.num_kv_heads <= 128 &&
                    al(a.key_cache) && al(a.value_cache) && al(a.query) && al(a.out) &&
                    (a.kv_block_stride * es) % 16 == 0 && (a.kv_head_stride * es) % 16 == 0 &&
                    (es == 1 || (tensor_map_stride(a.kv_block_stride) && tensor_map_stride(a.kv_head_stride))) &&
                    a.q_stride % 8 == 0 && tensor_map_stride(a.q_stride) && a.blocksparse_vert_stride <= 1 && a.out_lse == nullptr;
  if (!fits) return {nullptr, 0};
  return a.head_size <= 96 ? find_prefill_small(a.head_size, a.q_dtype, a.kv_dtype)
         : a.head_size <= 128 ? find_prefill_mid(a.head_size, a.q_dtype, a.kv_dtype)
                              : find_prefill_large(a.head_size, a.q_dtype, a.kv_dtype);
}

}  // namespace b200pa

extern "C" int b200pa_paged_attention_varlen_supported(const b200pa_attn_args* a) {
  return a != nullptr && a->num_heads > 0 && a->num_kv_heads > 0 && a->num_heads % a->num_kv_heads == 0 &&
         b200pa::find_prefill(b200pa::with_plain_strides(*a, 0)).fn != nullptr;
}

namespace b200pa {

// What a call is refused for, its decode rows among them; no more than CUDA errors can come behind it.
static int check_varlen(const b200pa_attn_args* a, const int32_t* query_start_loc, int32_t num_tokens, int32_t num_decodes,
                        PrefillKernelInfo* ki) {
  B200PA_CHECK_ARG(a->num_seqs >= 0 && a->num_heads > 0 && a->num_kv_heads > 0 && a->head_size > 0 &&
                       a->num_heads % a->num_kv_heads == 0,
                   "bad sizes: num_seqs=%d num_heads=%d num_kv_heads=%d head_size=%d", a->num_seqs,
                   a->num_heads, a->num_kv_heads, a->head_size);
  B200PA_CHECK_ARG(num_decodes >= 0 && num_decodes <= a->num_seqs && num_tokens >= num_decodes,
                   "bad counts: %d requests, %d decodes, %d tokens", a->num_seqs, num_decodes, num_tokens);
  if (a->num_seqs > num_decodes) {
    B200PA_CHECK_ARG(a->out && a->query && a->key_cache && a->value_cache && a->block_tables &&
                         a->seq_lens && query_start_loc,
                     "null tensor pointer");
    B200PA_CHECK_ARG(a->kv_dtype == B200PA_KV_AUTO || (a->k_scale && a->v_scale),
                     "fp8 kv cache needs k_scale and v_scale");
    B200PA_CHECK_ARG(a->max_num_blocks_per_seq > 0, "max_num_blocks_per_seq must be positive");
    *ki = find_prefill(*a);
    if (ki->fn == nullptr) {
      set_error("paged_attention_varlen: no kernel for head_size=%d block_size=%d q_dtype=%d kv_dtype=%d, "
                "or unaligned tensors",
                a->head_size, a->block_size, a->q_dtype, a->kv_dtype);
      return B200PA_EUNSUPPORTED;
    }
  }
  if (num_decodes == 0) return B200PA_OK;
  b200pa_attn_args d = *a;
  d.num_seqs = num_decodes;
  return attention_check(&d, false);
}

// `behind_write`: the launch in front on the stream is the KV write of the same step.
static int attention_varlen(const b200pa_attn_args* args, const int32_t* query_start_loc, int32_t num_tokens,
                            int32_t num_decodes, void* stream, bool behind_write) {
  B200PA_CHECK_ARG(args != nullptr, "args is NULL");
  const b200pa_attn_args plain = with_plain_strides(*args, num_tokens), *a = &plain;
  PrefillKernelInfo ki{nullptr, 0};
  if (const int bad = check_varlen(a, query_start_loc, num_tokens, num_decodes, &ki); bad != B200PA_OK) return bad;
  const int reqs = a->num_seqs - num_decodes;
  if (num_decodes > 0) {
    // the decode rows are the first rows of query and out: an ordinary decode batch
    b200pa_attn_args d = *a;
    d.num_seqs = num_decodes;
    const int rc = reqs > 0 ? attention_half_region(&d, stream, behind_write)
                   : behind_write ? attention_behind_write(&d, stream, false) : b200pa_paged_attention_v1(&d, stream);
    if (rc != B200PA_OK) return rc;
  }
  if (reqs == 0 || num_tokens == num_decodes) return B200PA_OK;  // (a tensor map has no empty dimension)

  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PrefillParams p{};
  p.out = a->out;
  p.q = a->query;
  p.kc = a->key_cache;
  p.vc = a->value_cache;
  p.alibi = a->alibi_slopes;
  p.k_scale = a->k_scale;
  p.v_scale = a->v_scale;
  p.q_stride = a->q_stride;
  p.kv_block_stride = a->kv_block_stride;
  p.kv_head_stride = a->kv_head_stride;
  p.num_heads = a->num_heads;
  p.num_tokens = num_tokens;
  p.num_kv_heads = a->num_kv_heads;
  p.group = a->num_heads / a->num_kv_heads;
  p.block_size = a->block_size;
  p.max_blocks_per_seq = a->max_num_blocks_per_seq;
  p.scale = a->scale;
  StreamRegion region{};
  if (stream_region(s, &region)) {  // (without one the keys of an item are not split)
    // (the second half: the first belongs to the decode launch, which may still be running)
    p.ws = region.ws + region.ws_bytes / 2;
    p.arrive = region.arrive + kArrivePerRegion / 2;
    p.ws_slots = int(std::min<int64_t>(int64_t(region.ws_bytes / 2) / ki.piece_bytes, kArrivePerRegion / 16));
    if (num_decodes == 0) {
      p.ws = region.ws;
      p.ws_slots = int(std::min<int64_t>(int64_t(region.ws_bytes) / ki.piece_bytes, kArrivePerRegion / 16));
    }
  }
  p.status = device_status_ptr();
  for (int r = num_decodes; r < a->num_seqs; r += kPrefillMaxReqs) {
    p.num_reqs = std::min(kPrefillMaxReqs, a->num_seqs - r);
    // nothing here depends on the decode launch: start where its CTAs have left, wait for it at the end
    p.late_wait = r == num_decodes && num_decodes > 0 ? 1 : 0;
    p.early = r == 0 && behind_write ? 1 : 0;
    p.block_tables = a->block_tables + int64_t(r) * a->max_num_blocks_per_seq;
    p.seq_lens = a->seq_lens + r;
    p.q_start = query_start_loc + r;
    p.sched = sched_words(s);
    if (p.sched == nullptr || p.status == nullptr) {
      set_error("could not resolve device-side scheduler/status words");
      return B200PA_ECUDA;
    }
    const cudaError_t e = ki.fn(p, sm_count(), s);
    count_launch();
    if (e != cudaSuccess) {
      set_error("prefill kernel launch failed: %s", cudaGetErrorString(e));
      return B200PA_ECUDA;
    }
  }
  return B200PA_OK;
}

}  // namespace b200pa

extern "C" int b200pa_paged_attention_varlen(const b200pa_attn_args* a, const int32_t* query_start_loc,
                                             int32_t num_tokens, int32_t num_decodes, void* stream) {
  return b200pa::attention_varlen(a, query_start_loc, num_tokens, num_decodes, stream, false);
}

extern "C" int b200pa_attention_step(const b200pa_cache_args* write, const b200pa_attn_args* a,
                                     const int32_t* query_start_loc, int32_t num_tokens, int32_t num_decodes,
                                     int32_t caller_scratch, void* stream) {
  using namespace b200pa;
  B200PA_CHECK_ARG(a != nullptr, "args is NULL");
  const b200pa_attn_args plain = with_plain_strides(*a, num_tokens);
  // (the write is launched only when the attention behind it will be)
  PrefillKernelInfo ki{nullptr, 0};
  const int bad = query_start_loc != nullptr ? check_varlen(&plain, query_start_loc, num_tokens, num_decodes, &ki)
                                             : attention_check(a, caller_scratch != 0);
  if (bad != B200PA_OK) return bad;
  bool behind_write = false;
  if (write != nullptr) {
    const int rc = b200pa_reshape_and_cache(write, stream);
    if (rc != B200PA_OK) return rc;
    behind_write = write->num_tokens > 0;
  }
  if (query_start_loc != nullptr)
    return attention_varlen(a, query_start_loc, num_tokens, num_decodes, stream, behind_write);
  if (behind_write) return attention_behind_write(a, stream, caller_scratch != 0);
  return caller_scratch != 0 ? b200pa_paged_attention_v2(a, stream) : b200pa_paged_attention_v1(a, stream);
}
