// PyTorch registration shim: the only file of the product that includes torch
// headers.  It unwraps tensors into the POD argument blocks of include/b200pa.h,
// sets the device guard, fetches the current stream, calls the C-ABI launcher
// and turns a non-zero return into a c10::Error (Python RuntimeError), like the
// reference's TORCH_CHECKs.
//
// Operator schemas are byte-for-byte those of the reference
// (csrc/torch_bindings.cpp:52-76, :687-704, :716-719).  The ops are always
// registered as torch.ops._C_b200.* / torch.ops._C_b200_cache_ops.*; on request
// (b200_claim_reference_names) also under the reference's own names
// (_C / _C_cache_ops), so code written against vllm._custom_ops runs unchanged.
#include <torch/csrc/autograd/python_variable.h>  // (Python.h comes first)

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/all.h>
#include <torch/library.h>

#include <cstdio>
#include <memory>
#include <optional>
#include <string>
#include <vector>

#include "../../include/b200pa.h"

namespace {

int dtype_code(at::ScalarType t, const char* what) {
  switch (t) {
    case at::ScalarType::Float: return B200PA_F32;
    case at::ScalarType::Half: return B200PA_F16;
    case at::ScalarType::BFloat16: return B200PA_BF16;
    default: TORCH_CHECK(false, "Unsupported input type of ", what, ": ", t);
  }
  return -1;
}

int kv_code(const std::string& s) {
  const int v = b200pa_kv_dtype_from_string(s.c_str());
  TORCH_CHECK(v >= 0, "Unsupported data type of kv cache: ", s);
  return v;
}

void check_rc(int rc) { TORCH_CHECK(rc == 0, "b200pa: ", b200pa_last_error()); }

void check_cuda(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
}

void fill_attn(b200pa_attn_args& a, torch::Tensor& out, torch::Tensor& query,
               torch::Tensor& key_cache, torch::Tensor& value_cache, int64_t num_kv_heads,
               double scale, torch::Tensor& block_tables, torch::Tensor& seq_lens,
               int64_t block_size, int64_t max_seq_len,
               const std::optional<torch::Tensor>& alibi_slopes, const std::string& kv_cache_dtype,
               torch::Tensor& k_scale, torch::Tensor& v_scale, int64_t tp_rank,
               int64_t bs_local, int64_t bs_vert, int64_t bs_block, int64_t bs_step) {
  check_cuda(out, "out");
  check_cuda(query, "query");
  check_cuda(key_cache, "key_cache");
  check_cuda(value_cache, "value_cache");
  check_cuda(block_tables, "block_tables");
  check_cuda(seq_lens, "seq_lens");
  TORCH_CHECK(query.dim() == 3, "query must be [num_seqs, num_heads, head_size]");
  TORCH_CHECK(out.is_contiguous(), "out must be contiguous");
  TORCH_CHECK(out.scalar_type() == query.scalar_type(), "out and query dtypes differ");
  TORCH_CHECK(query.stride(2) == 1 && query.stride(1) == query.size(2),
              "query heads must be contiguous");
  TORCH_CHECK(block_tables.scalar_type() == at::ScalarType::Int && block_tables.is_contiguous(),
              "block_tables must be a contiguous int32 tensor");
  TORCH_CHECK(seq_lens.scalar_type() == at::ScalarType::Int && seq_lens.is_contiguous(),
              "seq_lens must be a contiguous int32 tensor");
  TORCH_CHECK(key_cache.dim() == 5 && value_cache.dim() == 4, "caches must be 5-D (K) and 4-D (V)");
  std::memset(&a, 0, sizeof(a));
  a.q_dtype = dtype_code(query.scalar_type(), "kv cache");
  a.kv_dtype = kv_code(kv_cache_dtype);
  if (a.kv_dtype == B200PA_KV_AUTO) {
    TORCH_CHECK(key_cache.scalar_type() == query.scalar_type() &&
                    value_cache.scalar_type() == query.scalar_type(),
                "kv_cache_dtype 'auto' needs caches of the query dtype");
  } else {
    TORCH_CHECK(key_cache.element_size() == 1 && value_cache.element_size() == 1,
                "fp8 kv cache tensors must have 1-byte elements");
    TORCH_CHECK(k_scale.is_cuda() && v_scale.is_cuda() &&
                    k_scale.scalar_type() == at::ScalarType::Float &&
                    v_scale.scalar_type() == at::ScalarType::Float,
                "k_scale / v_scale must be float32 CUDA tensors");
  }
  a.out = out.data_ptr();
  a.query = query.data_ptr();
  a.key_cache = key_cache.data_ptr();
  a.value_cache = value_cache.data_ptr();
  a.block_tables = block_tables.data_ptr<int>();
  a.seq_lens = seq_lens.data_ptr<int>();
  if (alibi_slopes.has_value()) {
    TORCH_CHECK(alibi_slopes->scalar_type() == at::ScalarType::Float && alibi_slopes->is_cuda(),
                "alibi_slopes must be a float32 CUDA tensor");
    a.alibi_slopes = alibi_slopes->data_ptr<float>();
  }
  a.k_scale = k_scale.defined() && k_scale.is_cuda() ? static_cast<const float*>(k_scale.data_ptr()) : nullptr;
  a.v_scale = v_scale.defined() && v_scale.is_cuda() ? static_cast<const float*>(v_scale.data_ptr()) : nullptr;
  // (the stride of a dimension of size 1 means nothing, and may be 0)
  a.q_stride = query.size(0) == 1 ? query.size(1) * query.size(2) : query.stride(0);
  a.kv_block_stride = key_cache.size(0) == 1 ? key_cache.numel() : key_cache.stride(0);
  a.kv_head_stride = key_cache.stride(1);
  a.num_seqs = static_cast<int32_t>(query.size(0));
  a.num_heads = static_cast<int32_t>(query.size(1));
  a.num_kv_heads = static_cast<int32_t>(num_kv_heads);
  a.head_size = static_cast<int32_t>(query.size(2));
  a.block_size = static_cast<int32_t>(block_size);
  a.max_seq_len = static_cast<int32_t>(max_seq_len);
  a.max_num_blocks_per_seq = static_cast<int32_t>(block_tables.size(1));
  a.scale = static_cast<float>(scale);
  a.tp_rank = static_cast<int32_t>(tp_rank);
  a.blocksparse_local_blocks = static_cast<int32_t>(bs_local);
  a.blocksparse_vert_stride = static_cast<int32_t>(bs_vert);
  a.blocksparse_block_size = static_cast<int32_t>(bs_block);
  a.blocksparse_head_sliding_step = static_cast<int32_t>(bs_step);
}

void paged_attention_v1(torch::Tensor& out, torch::Tensor& query, torch::Tensor& key_cache,
                        torch::Tensor& value_cache, int64_t num_kv_heads, double scale,
                        torch::Tensor& block_tables, torch::Tensor& seq_lens, int64_t block_size,
                        int64_t max_seq_len, const std::optional<torch::Tensor>& alibi_slopes,
                        const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                        torch::Tensor& v_scale, const int64_t tp_rank,
                        const int64_t blocksparse_local_blocks,
                        const int64_t blocksparse_vert_stride,
                        const int64_t blocksparse_block_size,
                        const int64_t blocksparse_head_sliding_step) {
  b200pa_attn_args a;
  fill_attn(a, out, query, key_cache, value_cache, num_kv_heads, scale, block_tables, seq_lens,
            block_size, max_seq_len, alibi_slopes, kv_cache_dtype, k_scale, v_scale, tp_rank,
            blocksparse_local_blocks, blocksparse_vert_stride, blocksparse_block_size,
            blocksparse_head_sliding_step);
  const at::cuda::OptionalCUDAGuard device_guard(device_of(query));
  check_rc(b200pa_paged_attention_v1(&a, at::cuda::getCurrentCUDAStream().stream()));
}

// paged_attention_v1 that also returns the log-sum-exp of every (head, sequence), the
// quantity merge_attn_states needs to combine attention over disjoint token ranges.  Not
// an op of the reference: registered under the _C_b200 namespace only.
void paged_attention_with_lse(torch::Tensor& out, torch::Tensor& lse, torch::Tensor& query,
                              torch::Tensor& key_cache, torch::Tensor& value_cache,
                              int64_t num_kv_heads, double scale, torch::Tensor& block_tables,
                              torch::Tensor& seq_lens, int64_t block_size, int64_t max_seq_len,
                              const std::optional<torch::Tensor>& alibi_slopes,
                              const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                              torch::Tensor& v_scale) {
  b200pa_attn_args a;
  fill_attn(a, out, query, key_cache, value_cache, num_kv_heads, scale, block_tables, seq_lens,
            block_size, max_seq_len, alibi_slopes, kv_cache_dtype, k_scale, v_scale, 0, 0, 0, 64, 0);
  check_cuda(lse, "lse");
  TORCH_CHECK(lse.scalar_type() == at::ScalarType::Float && lse.is_contiguous() && lse.dim() == 2 &&
                  lse.size(0) == query.size(1) && lse.size(1) == query.size(0),
              "lse must be a contiguous float32 tensor [num_heads, num_seqs]");
  a.out_lse = lse.data_ptr<float>();
  const at::cuda::OptionalCUDAGuard device_guard(device_of(query));
  check_rc(b200pa_paged_attention_v1(&a, at::cuda::getCurrentCUDAStream().stream()));
}

void paged_attention_v2(torch::Tensor& out, torch::Tensor& exp_sums, torch::Tensor& max_logits,
                        torch::Tensor& tmp_out, torch::Tensor& query, torch::Tensor& key_cache,
                        torch::Tensor& value_cache, int64_t num_kv_heads, double scale,
                        torch::Tensor& block_tables, torch::Tensor& seq_lens, int64_t block_size,
                        int64_t max_seq_len, const std::optional<torch::Tensor>& alibi_slopes,
                        const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                        torch::Tensor& v_scale, const int64_t tp_rank,
                        const int64_t blocksparse_local_blocks,
                        const int64_t blocksparse_vert_stride,
                        const int64_t blocksparse_block_size,
                        const int64_t blocksparse_head_sliding_step) {
  b200pa_attn_args a;
  fill_attn(a, out, query, key_cache, value_cache, num_kv_heads, scale, block_tables, seq_lens,
            block_size, max_seq_len, alibi_slopes, kv_cache_dtype, k_scale, v_scale, tp_rank,
            blocksparse_local_blocks, blocksparse_vert_stride, blocksparse_block_size,
            blocksparse_head_sliding_step);
  check_cuda(exp_sums, "exp_sums");
  check_cuda(max_logits, "max_logits");
  check_cuda(tmp_out, "tmp_out");
  TORCH_CHECK(exp_sums.dim() == 3 && exp_sums.is_contiguous() && max_logits.is_contiguous() &&
                  tmp_out.is_contiguous(),
              "exp_sums / max_logits / tmp_out must be contiguous");
  TORCH_CHECK(exp_sums.scalar_type() == at::ScalarType::Float &&
                  max_logits.scalar_type() == at::ScalarType::Float &&
                  tmp_out.scalar_type() == query.scalar_type(),
              "exp_sums / max_logits must be float32 and tmp_out of the query dtype");
  TORCH_CHECK(max_logits.sizes() == exp_sums.sizes() && exp_sums.size(0) == query.size(0) &&
                  exp_sums.size(1) == query.size(1) && tmp_out.numel() == exp_sums.numel() * query.size(2),
              "v2 scratch tensors have inconsistent shapes");
  a.exp_sums = exp_sums.data_ptr<float>();
  a.max_logits = max_logits.data_ptr<float>();
  a.tmp_out = tmp_out.data_ptr();
  a.max_num_partitions = static_cast<int32_t>(exp_sums.size(2));
  const at::cuda::OptionalCUDAGuard device_guard(device_of(query));
  check_rc(b200pa_paged_attention_v2(&a, at::cuda::getCurrentCUDAStream().stream()));
}

// Attention of a step whose requests bring several query rows (not an op of the reference).
// False: no kernel for this shape, nothing was launched.
bool paged_attention_varlen(torch::Tensor& out, torch::Tensor& query, torch::Tensor& key_cache,
                            torch::Tensor& value_cache, int64_t num_kv_heads, double scale,
                            torch::Tensor& block_tables, torch::Tensor& seq_lens,
                            torch::Tensor& query_start_loc, int64_t num_decodes, int64_t block_size,
                            int64_t max_seq_len, const std::optional<torch::Tensor>& alibi_slopes,
                            const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                            torch::Tensor& v_scale) {
  b200pa_attn_args a;
  fill_attn(a, out, query, key_cache, value_cache, num_kv_heads, scale, block_tables, seq_lens,
            block_size, max_seq_len, alibi_slopes, kv_cache_dtype, k_scale, v_scale, 0, 0, 0, 64, 0);
  TORCH_CHECK(query_start_loc.is_cuda() && query_start_loc.scalar_type() == at::ScalarType::Int &&
                  query_start_loc.is_contiguous() && query_start_loc.numel() == seq_lens.numel() + 1,
              "query_start_loc must be a contiguous int32 CUDA tensor [num_requests + 1]");
  a.num_seqs = static_cast<int32_t>(seq_lens.size(0));
  const at::cuda::OptionalCUDAGuard device_guard(device_of(query));
  const int rc = b200pa_paged_attention_varlen(&a, query_start_loc.data_ptr<int>(),
                                               static_cast<int32_t>(query.size(0)),
                                               static_cast<int32_t>(num_decodes),
                                               at::cuda::getCurrentCUDAStream().stream());
  if (rc == B200PA_EUNSUPPORTED) return false;
  check_rc(rc);
  return true;
}

void fill_cache(b200pa_cache_args& a, torch::Tensor& key, torch::Tensor& value,
                torch::Tensor& key_cache, torch::Tensor& value_cache, torch::Tensor& slot_mapping,
                const std::string& kv_cache_dtype, torch::Tensor& k_scale, torch::Tensor& v_scale) {
  check_cuda(key, "key");
  check_cuda(value, "value");
  check_cuda(key_cache, "key_cache");
  check_cuda(value_cache, "value_cache");
  check_cuda(slot_mapping, "slot_mapping");
  TORCH_CHECK(key.dim() == 3 && value.dim() == 3, "key/value must be [num_tokens, num_heads, head_size]");
  TORCH_CHECK(key.stride(2) == 1 && key.stride(1) == key.size(2) && value.stride(2) == 1 &&
                  value.stride(1) == value.size(2),
              "key/value heads must be contiguous");
  TORCH_CHECK(slot_mapping.scalar_type() == at::ScalarType::Long && slot_mapping.is_contiguous(),
              "slot_mapping must be a contiguous int64 tensor");
  std::memset(&a, 0, sizeof(a));
  a.in_dtype = dtype_code(key.scalar_type(), "kv cache");
  TORCH_CHECK(value.scalar_type() == key.scalar_type(), "key and value dtypes differ");
  a.kv_dtype = kv_code(kv_cache_dtype);
  if (a.kv_dtype == B200PA_KV_AUTO) {
    TORCH_CHECK(key_cache.scalar_type() == key.scalar_type() &&
                    value_cache.scalar_type() == key.scalar_type(),
                "kv_cache_dtype 'auto' needs caches of the key dtype");
  } else {
    TORCH_CHECK(key_cache.element_size() == 1 && value_cache.element_size() == 1,
                "fp8 kv cache tensors must have 1-byte elements");
    TORCH_CHECK(k_scale.is_cuda() && v_scale.is_cuda() &&
                    k_scale.scalar_type() == at::ScalarType::Float &&
                    v_scale.scalar_type() == at::ScalarType::Float,
                "k_scale / v_scale must be float32 CUDA tensors");
  }
  a.key = key.data_ptr();
  a.value = value.data_ptr();
  a.key_cache = key_cache.data_ptr();
  a.value_cache = value_cache.data_ptr();
  a.slot_mapping = slot_mapping.data_ptr<int64_t>();
  a.k_scale = k_scale.defined() && k_scale.is_cuda() ? static_cast<const float*>(k_scale.data_ptr()) : nullptr;
  a.v_scale = v_scale.defined() && v_scale.is_cuda() ? static_cast<const float*>(v_scale.data_ptr()) : nullptr;
  a.key_stride = key.stride(0);
  a.value_stride = value.stride(0);
  a.num_tokens = static_cast<int32_t>(slot_mapping.size(0));
  a.num_heads = static_cast<int32_t>(key.size(1));
  a.head_size = static_cast<int32_t>(key.size(2));
}

void reshape_and_cache(torch::Tensor& key, torch::Tensor& value, torch::Tensor& key_cache,
                       torch::Tensor& value_cache, torch::Tensor& slot_mapping,
                       const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                       torch::Tensor& v_scale) {
  b200pa_cache_args a;
  fill_cache(a, key, value, key_cache, value_cache, slot_mapping, kv_cache_dtype, k_scale, v_scale);
  TORCH_CHECK(key_cache.dim() == 5 && value_cache.dim() == 4,
              "key_cache must be [num_blocks, num_heads, head_size/x, block_size, x] and "
              "value_cache [num_blocks, num_heads, head_size, block_size]");
  TORCH_CHECK(key_cache.is_contiguous() && value_cache.is_contiguous(),
              "reshape_and_cache needs contiguous caches");
  a.block_size = static_cast<int32_t>(key_cache.size(3));
  a.x = static_cast<int32_t>(key_cache.size(4));
  const at::cuda::OptionalCUDAGuard device_guard(device_of(key));
  check_rc(b200pa_reshape_and_cache(&a, at::cuda::getCurrentCUDAStream().stream()));
}

void reshape_and_cache_flash(torch::Tensor& key, torch::Tensor& value, torch::Tensor& key_cache,
                             torch::Tensor& value_cache, torch::Tensor& slot_mapping,
                             const std::string& kv_cache_dtype, torch::Tensor& k_scale,
                             torch::Tensor& v_scale) {
  b200pa_cache_args a;
  fill_cache(a, key, value, key_cache, value_cache, slot_mapping, kv_cache_dtype, k_scale, v_scale);
  TORCH_CHECK(key_cache.dim() == 4 && value_cache.dim() == 4,
              "caches must be [num_blocks, block_size, num_heads, head_size] (possibly strided)");
  TORCH_CHECK(key_cache.stride(0) == value_cache.stride(0));
  TORCH_CHECK(key_cache.stride(3) == 1 && value_cache.stride(3) == 1,
              "the head_size dimension of the caches must be contiguous");
  a.block_size = static_cast<int32_t>(key_cache.size(1));
  a.block_stride = key_cache.stride(0);
  a.page_stride = key_cache.stride(1);
  a.head_stride = key_cache.stride(2);
  const at::cuda::OptionalCUDAGuard device_guard(device_of(key));
  check_rc(b200pa_reshape_and_cache_flash(&a, at::cuda::getCurrentCUDAStream().stream()));
}

void convert_fp8(torch::Tensor& dst_cache, torch::Tensor& src_cache, const double scale,
                 const std::string& kv_cache_dtype) {
  TORCH_CHECK(src_cache.is_cuda(), "src must be on a GPU");
  TORCH_CHECK(dst_cache.is_cuda(), "dst must be on a GPU");
  TORCH_CHECK(src_cache.device() == dst_cache.device(), "src and dst must be on the same GPU");
  TORCH_CHECK(src_cache.is_contiguous() && dst_cache.is_contiguous() &&
                  src_cache.numel() == dst_cache.numel(),
              "convert_fp8 needs contiguous tensors of equal size");
  int kv;
  if (kv_cache_dtype == "auto" || kv_cache_dtype == "fp8" || kv_cache_dtype == "fp8_e4m3") {
    kv = B200PA_KV_FP8_E4M3;
  } else if (kv_cache_dtype == "fp8_e5m2") {
    kv = B200PA_KV_FP8_E5M2;
  } else {
    TORCH_CHECK(false, "Unsupported data type: ", kv_cache_dtype);
  }
  const bool to_fp8 = dst_cache.element_size() == 1;
  TORCH_CHECK(to_fp8 != (src_cache.element_size() == 1),
              "exactly one of src / dst must be a 1-byte (fp8) tensor");
  const int wide = dtype_code(to_fp8 ? src_cache.scalar_type() : dst_cache.scalar_type(), "convert_fp8");
  const at::cuda::OptionalCUDAGuard device_guard(src_cache.device());
  check_rc(b200pa_convert_fp8(dst_cache.data_ptr(), src_cache.data_ptr(), src_cache.numel(),
                              static_cast<float>(scale), wide, kv, to_fp8 ? 1 : 0,
                              at::cuda::getCurrentCUDAStream().stream()));
}

void merge_attn_states(torch::Tensor& output, std::optional<torch::Tensor> output_lse,
                       const torch::Tensor& prefix_output, const torch::Tensor& prefix_lse,
                       const torch::Tensor& suffix_output, const torch::Tensor& suffix_lse) {
  check_cuda(output, "output");
  TORCH_CHECK(output.dim() == 3, "output must be [num_tokens, num_heads, head_size]");
  const int dt = [&]() -> int {
    switch (output.scalar_type()) {
      case at::ScalarType::Float: return B200PA_F32;
      case at::ScalarType::Half: return B200PA_F16;
      case at::ScalarType::BFloat16: return B200PA_BF16;
      default: TORCH_CHECK(false, "Unsupported data type of O: ", output.scalar_type());
    }
    return -1;
  }();
  const int64_t head_size = output.size(2);
  TORCH_CHECK(output.stride(-2) == head_size && output.stride(-1) == 1,
              "output heads must be contiguous");
  TORCH_CHECK(prefix_output.stride(-2) == head_size && prefix_output.stride(-1) == 1,
              "prefix_output heads must be contiguous");
  TORCH_CHECK(suffix_output.stride(-2) == head_size && suffix_output.stride(-1) == 1,
              "suffix_output heads must be contiguous");
  TORCH_CHECK(output.is_contiguous() && prefix_output.is_contiguous() &&
                  suffix_output.is_contiguous() && prefix_lse.is_contiguous() &&
                  suffix_lse.is_contiguous(),
              "merge_attn_states needs contiguous tensors");
  TORCH_CHECK(prefix_output.scalar_type() == output.scalar_type() &&
                  suffix_output.scalar_type() == output.scalar_type(),
              "prefix/suffix/output dtypes differ");
  TORCH_CHECK(prefix_lse.scalar_type() == at::ScalarType::Float &&
                  suffix_lse.scalar_type() == at::ScalarType::Float,
              "lse tensors must be float32");
  float* olse = nullptr;
  if (output_lse.has_value()) {
    TORCH_CHECK(output_lse->scalar_type() == at::ScalarType::Float && output_lse->is_contiguous(),
                "output_lse must be a contiguous float32 tensor");
    olse = output_lse->data_ptr<float>();
  }
  const at::cuda::OptionalCUDAGuard device_guard(device_of(output));
  check_rc(b200pa_merge_attn_states(output.data_ptr(), olse, prefix_output.data_ptr(),
                                    prefix_lse.data_ptr<float>(), suffix_output.data_ptr(),
                                    suffix_lse.data_ptr<float>(), output.size(0),
                                    static_cast<int32_t>(output.size(1)),
                                    static_cast<int32_t>(head_size), dt,
                                    at::cuda::getCurrentCUDAStream().stream()));
}

void copy_blocks(std::vector<torch::Tensor> const& key_caches,
                 std::vector<torch::Tensor> const& value_caches,
                 const torch::Tensor& block_mapping) {
  const size_t num_layers = key_caches.size();
  TORCH_CHECK(num_layers == value_caches.size());
  if (num_layers == 0) return;
  TORCH_CHECK(key_caches[0].is_cuda());
  TORCH_CHECK(block_mapping.is_cuda() && block_mapping.scalar_type() == at::ScalarType::Long &&
                  block_mapping.is_contiguous() && block_mapping.dim() == 2 &&
                  block_mapping.size(1) == 2,
              "block_mapping must be a contiguous int64 CUDA tensor of shape [num_pairs, 2]");
  std::vector<void*> kp(num_layers), vp(num_layers);
  for (size_t i = 0; i < num_layers; ++i) {
    kp[i] = key_caches[i].data_ptr();
    vp[i] = value_caches[i].data_ptr();
  }
  const int64_t block_bytes = key_caches[0][0].numel() * key_caches[0].element_size();
  const at::cuda::OptionalCUDAGuard device_guard(key_caches[0].device());
  check_rc(b200pa_copy_blocks(kp.data(), vp.data(), static_cast<int32_t>(num_layers),
                              block_mapping.data_ptr<int64_t>(), block_mapping.size(0),
                              block_bytes, at::cuda::getCurrentCUDAStream().stream()));
}

void swap_blocks(torch::Tensor& src, torch::Tensor& dst, const torch::Tensor& block_mapping) {
  const bool sc = src.is_cuda(), dc = dst.is_cuda();
  if (sc && dc) {
    TORCH_CHECK(src.device() == dst.device(), "src and dst must be on the same GPU");
  } else {
    TORCH_CHECK((sc && dst.is_cpu()) || (src.is_cpu() && dc), "Invalid device combination");
  }
  TORCH_CHECK(block_mapping.device().is_cpu(), "block_mapping must be on CPU");
  TORCH_CHECK(block_mapping.scalar_type() == at::ScalarType::Long && block_mapping.dim() == 2 &&
                  block_mapping.size(1) == 2,
              "block_mapping must be an int64 tensor of shape [num_pairs, 2]");
  const torch::Tensor bm = block_mapping.contiguous();
  // the stride, not numel, so that padded blocks are copied whole (as the reference does)
  const int64_t block_bytes = src.element_size() * src.stride(0);
  const at::cuda::OptionalCUDAGuard device_guard(sc ? src.device() : dst.device());
  check_rc(b200pa_swap_blocks(src.data_ptr(), dst.data_ptr(), bm.data_ptr<int64_t>(), bm.size(0),
                              block_bytes, at::cuda::getCurrentCUDAStream().stream()));
}

constexpr const char* kMergeSchema =
    "merge_attn_states("
    "    Tensor! output,"
    "    Tensor!? output_lse,"
    "    Tensor prefix_output,"
    "    Tensor prefix_lse,"
    "    Tensor suffix_output,"
    "    Tensor suffix_lse) -> ()";
constexpr const char* kSwapSchema = "swap_blocks(Tensor src, Tensor! dst, Tensor block_mapping) -> ()";
constexpr const char* kCopySchema =
    "copy_blocks(Tensor(a!)[] key_caches, Tensor[](b!) value_caches, "
    "Tensor block_mapping) -> ()";
constexpr const char* kV1Schema =
    "paged_attention_v1("
    "    Tensor! out, Tensor query, Tensor key_cache,"
    "    Tensor value_cache, int num_kv_heads, float scale,"
    "    Tensor block_tables, Tensor seq_lens, int block_size,"
    "    int max_seq_len, Tensor? alibi_slopes,"
    "    str kv_cache_dtype, Tensor k_scale, Tensor v_scale,"
    "    int tp_rank, int blocksparse_local_blocks,"
    "    int blocksparse_vert_stride, int blocksparse_block_size,"
    "    int blocksparse_head_sliding_step) -> ()";
constexpr const char* kV2Schema =
    "paged_attention_v2("
    "    Tensor! out, Tensor! exp_sums, Tensor! max_logits,"
    "    Tensor! tmp_out, Tensor query, Tensor key_cache,"
    "    Tensor value_cache, int num_kv_heads, float scale,"
    "    Tensor block_tables, Tensor seq_lens, int block_size,"
    "    int max_seq_len, Tensor? alibi_slopes,"
    "    str kv_cache_dtype, Tensor k_scale, Tensor v_scale,"
    "    int tp_rank, int blocksparse_local_blocks,"
    "    int blocksparse_vert_stride, int blocksparse_block_size,"
    "    int blocksparse_head_sliding_step) -> ()";
constexpr const char* kReshapeSchema =
    "reshape_and_cache(Tensor key, Tensor value,"
    "                  Tensor! key_cache, Tensor! value_cache,"
    "                  Tensor slot_mapping,"
    "                  str kv_cache_dtype,"
    "                  Tensor k_scale, Tensor v_scale) -> ()";
constexpr const char* kReshapeFlashSchema =
    "reshape_and_cache_flash(Tensor key, Tensor value,"
    "                        Tensor! key_cache,"
    "                        Tensor! value_cache,"
    "                        Tensor slot_mapping,"
    "                        str kv_cache_dtype,"
    "                        Tensor k_scale, Tensor v_scale) -> ()";
constexpr const char* kConvertSchema =
    "convert_fp8(Tensor! dst_cache, Tensor src_cache, float scale, "
    "str kv_cache_dtype) -> ()";

bool op_exists(const char* qualified) {
  return c10::Dispatcher::singleton().findSchema({qualified, ""}).has_value();
}

}  // namespace

TORCH_LIBRARY(_C_b200, ops) {
  ops.def(kV1Schema);
  ops.impl("paged_attention_v1", torch::kCUDA, &paged_attention_v1);
  ops.def(kV2Schema);
  ops.impl("paged_attention_v2", torch::kCUDA, &paged_attention_v2);
  ops.def(kMergeSchema);
  ops.impl("merge_attn_states", torch::kCUDA, &merge_attn_states);
  ops.def(
      "paged_attention_with_lse(Tensor! out, Tensor! lse, Tensor query, Tensor key_cache,"
      " Tensor value_cache, int num_kv_heads, float scale, Tensor block_tables, Tensor seq_lens,"
      " int block_size, int max_seq_len, Tensor? alibi_slopes, str kv_cache_dtype,"
      " Tensor k_scale, Tensor v_scale) -> ()");
  ops.impl("paged_attention_with_lse", torch::kCUDA, &paged_attention_with_lse);
}

// (see b200pa_paged_attention_varlen)
TORCH_LIBRARY_FRAGMENT(_C_b200, ops) {
  ops.def(
      "paged_attention_varlen(Tensor! out, Tensor query, Tensor key_cache, Tensor value_cache,"
      " int num_kv_heads, float scale, Tensor block_tables, Tensor seq_lens, Tensor query_start_loc,"
      " int num_decodes, int block_size, int max_seq_len, Tensor? alibi_slopes, str kv_cache_dtype,"
      " Tensor k_scale, Tensor v_scale) -> bool");
  ops.impl("paged_attention_varlen", torch::kCUDA, &paged_attention_varlen);
}

TORCH_LIBRARY(_C_b200_cache_ops, cache_ops) {
  cache_ops.def(kSwapSchema);
  cache_ops.impl("swap_blocks", torch::kCUDA, &swap_blocks);
  cache_ops.def(kCopySchema);
  cache_ops.impl("copy_blocks", torch::kCUDA, &copy_blocks);
  cache_ops.def(kReshapeSchema);
  cache_ops.impl("reshape_and_cache", torch::kCUDA, &reshape_and_cache);
  cache_ops.def(kReshapeFlashSchema);
  cache_ops.impl("reshape_and_cache_flash", torch::kCUDA, &reshape_and_cache_flash);
  cache_ops.def(kConvertSchema);
  cache_ops.impl("convert_fp8", torch::kCUDA, &convert_fp8);
}

// The reference's own operator names (_C / _C_cache_ops) are claimed on request only, never
// while this library loads: if they were defined here first, a vLLM `_C` extension imported
// afterwards would fail on the duplicate definitions.  A stand-alone user (the reference's
// own tests and benchmarks run without vLLM's extension) asks for them once with
// vllm_b200.claim_reference_names(); names that somebody has defined already are left alone.
// Returns how many names were claimed by this call, or -1 with `err` filled in.
extern "C" int b200_claim_reference_names(char* err, int err_len) {
  static std::vector<std::unique_ptr<torch::Library>> keep;  // registrations live as long as these
  try {
    int n = 0;
    auto ops = std::make_unique<torch::Library>(torch::Library::FRAGMENT, "_C", std::nullopt,
                                                __FILE__, __LINE__);
    auto cache_ops = std::make_unique<torch::Library>(torch::Library::FRAGMENT, "_C_cache_ops",
                                                      std::nullopt, __FILE__, __LINE__);
    if (!op_exists("_C::paged_attention_v1")) {
      ops->def(kV1Schema);
      ops->impl("paged_attention_v1", torch::kCUDA, &paged_attention_v1);
      ++n;
    }
    if (!op_exists("_C::paged_attention_v2")) {
      ops->def(kV2Schema);
      ops->impl("paged_attention_v2", torch::kCUDA, &paged_attention_v2);
      ++n;
    }
    if (!op_exists("_C::merge_attn_states")) {
      ops->def(kMergeSchema);
      ops->impl("merge_attn_states", torch::kCUDA, &merge_attn_states);
      ++n;
    }
    if (!op_exists("_C_cache_ops::reshape_and_cache")) {
      cache_ops->def(kReshapeSchema);
      cache_ops->impl("reshape_and_cache", torch::kCUDA, &reshape_and_cache);
      ++n;
    }
    if (!op_exists("_C_cache_ops::reshape_and_cache_flash")) {
      cache_ops->def(kReshapeFlashSchema);
      cache_ops->impl("reshape_and_cache_flash", torch::kCUDA, &reshape_and_cache_flash);
      ++n;
    }
    if (!op_exists("_C_cache_ops::swap_blocks")) {
      cache_ops->def(kSwapSchema);
      cache_ops->impl("swap_blocks", torch::kCUDA, &swap_blocks);
      ++n;
    }
    if (!op_exists("_C_cache_ops::copy_blocks")) {
      cache_ops->def(kCopySchema);
      cache_ops->impl("copy_blocks", torch::kCUDA, &copy_blocks);
      ++n;
    }
    if (!op_exists("_C_cache_ops::convert_fp8")) {
      cache_ops->def(kConvertSchema);
      cache_ops->impl("convert_fp8", torch::kCUDA, &convert_fp8);
      ++n;
    }
    keep.push_back(std::move(ops));
    keep.push_back(std::move(cache_ops));
    return n;
  } catch (const std::exception& e) {
    if (err != nullptr && err_len > 0) snprintf(err, size_t(err_len), "%s", e.what());
    return -1;
  }
}

// ------------------------------------------------------------------ direct Python bindings
// A call through torch.ops costs 4-8 us of host time with arguments as many as these (boxing, schema
// matching, dispatch), more than the small launches take on the GPU.  The module below binds the
// same functions directly.  Every function returns True when it has done the work, and False when
// the call is not the plain case - tensor subclasses, tracing or dispatch modes, profiling, autograd,
// anything that a check objects to: the wrapper then goes through torch.ops, which handles it or
// raises.
namespace {

// The calling thread's state allows a call that the dispatcher does not see: no modes, no profiler, and no
// dispatch keys beyond the usual ones (tracing, functionalization and the function transforms add theirs).
bool plain_state() {
  const c10::DispatchKeySet more = c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set;
  return more.empty() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !at::impl::torch_function_mode_enabled() && !at::hasCallbacks();
}

bool plain_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && !t.key_set().has(c10::DispatchKey::Python) &&
         !(t.requires_grad() && c10::GradMode::is_enabled());
}

// Reads positional arguments in order; `ok` turns false at the first one that is not plain.
struct Args {
  PyObject* const* a;
  Py_ssize_t n, i = 0;
  bool ok = true;
  PyObject* next() {
    if (i >= n) ok = false;
    return ok ? a[i++] : nullptr;
  }
  at::Tensor tensor() {
    PyObject* o = next();
    if (o == nullptr || !plain_tensor(o)) return ok = false, at::Tensor();
    return THPVariable_Unpack(o);
  }
  std::optional<at::Tensor> optional_tensor() {
    PyObject* o = next();
    if (o == nullptr || o == Py_None) return std::nullopt;
    if (!plain_tensor(o)) return ok = false, std::nullopt;
    return THPVariable_Unpack(o);
  }
  int64_t integer() {
    PyObject* o = next();
    if (o == nullptr || !PyLong_Check(o)) return ok = false, 0;
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) PyErr_Clear(), ok = false;
    return v;
  }
  double real() {
    PyObject* o = next();
    if (o == nullptr || !PyFloat_Check(o)) return ok = false, 0.0;
    return PyFloat_AS_DOUBLE(o);
  }
  std::string text() {
    PyObject* o = next();
    if (o == nullptr || !PyUnicode_Check(o)) return ok = false, std::string();
    Py_ssize_t len = 0;
    const char* s = PyUnicode_AsUTF8AndSize(o, &len);
    if (s == nullptr) return PyErr_Clear(), ok = false, std::string();
    return std::string(s, size_t(len));
  }
};

template <typename F>
PyObject* direct(Args& in, F&& call) {
  bool done = false;
  if (in.ok && in.i == in.n) {
    PyThreadState* ts = PyEval_SaveThread();
    try {
      done = call();
    } catch (...) {
      // the wrapper's call through torch.ops raises it again, with everything a caller expects
      (void)cudaGetLastError();
    }
    PyEval_RestoreThread(ts);
  }
  return PyBool_FromLong(done);
}

PyObject* py_paged_attention(PyObject* const* a, Py_ssize_t n, bool v2) {
  if (!plain_state()) Py_RETURN_FALSE;
  Args in{a, n};
  at::Tensor out = in.tensor(), es, ml, tmp;
  if (v2) {
    es = in.tensor();
    ml = in.tensor();
    tmp = in.tensor();
  }
  at::Tensor q = in.tensor(), kc = in.tensor(), vc = in.tensor();
  const int64_t hk = in.integer();
  const double scale = in.real();
  at::Tensor bt = in.tensor(), sl = in.tensor();
  const int64_t bs = in.integer(), max_len = in.integer();
  const auto alibi = in.optional_tensor();
  const std::string kv = in.text();
  at::Tensor ks = in.tensor(), vs = in.tensor();
  const int64_t tp = in.integer(), b0 = in.integer(), b1 = in.integer(), b2 = in.integer(), b3 = in.integer();
  return direct(in, [&] {
    if (v2)
      paged_attention_v2(out, es, ml, tmp, q, kc, vc, hk, scale, bt, sl, bs, max_len, alibi, kv, ks, vs, tp, b0,
                         b1, b2, b3);
    else
      paged_attention_v1(out, q, kc, vc, hk, scale, bt, sl, bs, max_len, alibi, kv, ks, vs, tp, b0, b1, b2, b3);
    return true;
  });
}
PyObject* py_v1(PyObject*, PyObject* const* a, Py_ssize_t n) { return py_paged_attention(a, n, false); }
PyObject* py_v2(PyObject*, PyObject* const* a, Py_ssize_t n) { return py_paged_attention(a, n, true); }

PyObject* py_write(PyObject* const* a, Py_ssize_t n, bool flash) {
  if (!plain_state()) Py_RETURN_FALSE;
  Args in{a, n};
  at::Tensor k = in.tensor(), v = in.tensor(), kc = in.tensor(), vc = in.tensor(), slots = in.tensor();
  const std::string kv = in.text();
  at::Tensor ks = in.tensor(), vs = in.tensor();
  return direct(in, [&] {
    if (flash) reshape_and_cache_flash(k, v, kc, vc, slots, kv, ks, vs);
    else reshape_and_cache(k, v, kc, vc, slots, kv, ks, vs);
    return true;
  });
}
PyObject* py_write_x(PyObject*, PyObject* const* a, Py_ssize_t n) { return py_write(a, n, false); }
PyObject* py_write_flash(PyObject*, PyObject* const* a, Py_ssize_t n) { return py_write(a, n, true); }

// One attention layer of an engine step: KV write, then attention, straight from the tensors that
// the engine hands over (no views, no copies, no scratch tensors where the library's workspace does).
PyObject* py_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!plain_state()) Py_RETURN_FALSE;
  Args in{a, n};
  at::Tensor out = in.tensor(), q = in.tensor(), k = in.tensor(), v = in.tensor(), cache = in.tensor();
  at::Tensor bt = in.tensor(), sl = in.tensor(), slots = in.tensor(), qsl = in.tensor();
  at::Tensor ks = in.tensor(), vs = in.tensor();
  const auto alibi = in.optional_tensor();
  const int64_t tokens = in.integer(), decodes = in.integer(), max_q = in.integer(), max_len = in.integer();
  const int64_t H = in.integer(), HK = in.integer(), D = in.integer();
  const double scale = in.real();
  const std::string kv = in.text();
  const int64_t write = in.integer(), prefer_v1 = in.integer();
  return direct(in, [&]() -> bool {
    using at::ScalarType;
    const auto type = q.scalar_type();
    const bool fp8 = kv != "auto";
    // rows of q, k, v: heads and head dimensions contiguous
    auto rows = [&](const at::Tensor& t, int64_t heads) {
      return t.dim() == 3 && t.size(0) >= tokens && t.size(1) == heads && t.size(2) == D && t.stride(2) == 1 &&
             t.stride(1) == D && t.scalar_type() == type;
    };
    if (type != ScalarType::BFloat16 && type != ScalarType::Half) return false;
    if (tokens <= 0 || H <= 0 || HK <= 0 || D <= 0 || H % HK != 0) return false;
    if (!rows(q, H) || !rows(k, HK) || !rows(v, HK)) return false;
    if (!out.is_contiguous() || out.numel() < tokens * H * D || out.scalar_type() != type) return false;
    if (cache.dim() != 3 || cache.size(0) != 2 || !cache.is_contiguous() || cache.size(2) % (HK * D) != 0)
      return false;
    if (fp8 ? cache.element_size() != 1 : cache.scalar_type() != type) return false;
    const int64_t B = cache.size(2) / (HK * D), x = 16 / cache.element_size();
    if (B <= 0 || D % x != 0) return false;
    const int64_t reqs = sl.numel();
    if (bt.dim() != 2 || bt.size(0) < reqs || !bt.is_contiguous() || bt.scalar_type() != ScalarType::Int ||
        !sl.is_contiguous() || sl.scalar_type() != ScalarType::Int || slots.dim() != 1 ||
        !slots.is_contiguous() || slots.numel() < tokens || slots.scalar_type() != ScalarType::Long ||
        ks.scalar_type() != ScalarType::Float || vs.scalar_type() != ScalarType::Float)
      return false;
    if (alibi.has_value() && (alibi->scalar_type() != ScalarType::Float || alibi->numel() != H)) return false;
    if (max_q == 1) {
      if (reqs < tokens) return false;
    } else if (decodes < 0 || decodes > reqs || !qsl.is_contiguous() || qsl.scalar_type() != ScalarType::Int ||
               qsl.numel() != reqs + 1) {
      return false;
    }
    const auto dev = q.device();
    for (const at::Tensor* t : {&out, &k, &v, &cache, &bt, &sl, &slots, &qsl, &ks, &vs})
      if (t->device() != dev) return false;

    char* base = static_cast<char*>(cache.data_ptr());
    char* vbase = base + cache.stride(0) * cache.element_size();
    const int in_type = type == ScalarType::BFloat16 ? B200PA_BF16 : B200PA_F16;
    const int kv_type = kv_code(kv);
    const at::cuda::OptionalCUDAGuard device_guard(dev);
    void* stream = at::cuda::getCurrentCUDAStream().stream();
    b200pa_attn_args p;
    std::memset(&p, 0, sizeof(p));
    p.q_dtype = in_type;
    p.kv_dtype = kv_type;
    p.out = out.data_ptr();
    p.query = q.data_ptr();
    p.key_cache = base;
    p.value_cache = vbase;
    p.block_tables = bt.data_ptr<int>();
    p.seq_lens = sl.data_ptr<int>();
    p.alibi_slopes = alibi.has_value() ? alibi->data_ptr<float>() : nullptr;
    p.k_scale = ks.data_ptr<float>();
    p.v_scale = vs.data_ptr<float>();
    p.q_stride = tokens == 1 ? H * D : q.stride(0);
    p.kv_block_stride = HK * D * B;
    p.kv_head_stride = D * B;
    p.num_seqs = static_cast<int32_t>(max_q == 1 ? tokens : reqs);
    p.num_heads = static_cast<int32_t>(H);
    p.num_kv_heads = static_cast<int32_t>(HK);
    p.head_size = static_cast<int32_t>(D);
    p.block_size = static_cast<int32_t>(B);
    p.max_seq_len = static_cast<int32_t>(max_len);
    p.max_num_blocks_per_seq = static_cast<int32_t>(bt.size(1));
    p.scale = static_cast<float>(scale);
    p.blocksparse_block_size = 64;
    // (nothing may be done before it is clear that everything can be: the caller would do it again)
    if (max_q > 1 && decodes < reqs && !b200pa_paged_attention_varlen_supported(&p)) return false;
    b200pa_cache_args c;
    std::memset(&c, 0, sizeof(c));
    if (write) {
      c.in_dtype = in_type;
      c.kv_dtype = kv_type;
      c.key = k.data_ptr();
      c.value = v.data_ptr();
      c.key_cache = base;
      c.value_cache = vbase;
      c.slot_mapping = slots.data_ptr<int64_t>();
      c.k_scale = ks.data_ptr<float>();
      c.v_scale = vs.data_ptr<float>();
      c.key_stride = k.stride(0);
      c.value_stride = v.stride(0);
      c.num_tokens = static_cast<int32_t>(tokens);
      c.num_heads = static_cast<int32_t>(HK);
      c.head_size = static_cast<int32_t>(D);
      c.block_size = static_cast<int32_t>(B);
      c.x = static_cast<int32_t>(x);
    }
    auto run = [&](const int* starts, bool caller_scratch) {
      check_rc(b200pa_attention_step(write ? &c : nullptr, &p, starts, static_cast<int32_t>(tokens),
                                     static_cast<int32_t>(decodes), caller_scratch, stream));
    };
    if (max_q > 1) {
      run(qsl.data_ptr<int>(), false);
      return true;
    }
    // v1 also when the partials of v2 fit the library's own workspace, which saves the scratch allocation
    const int64_t parts = (max_len + 511) / 512, rows_n = tokens * H;
    const bool use_v1 =
        prefer_v1 != 0 || rows_n * parts * (8 + 2 * D) <= b200pa_stream_workspace_bytes() - 1024;
    if (use_v1) {
      run(nullptr, false);
      return true;
    }
    const int64_t stat = (rows_n * parts * 4 + 255) & ~int64_t(255);
    const at::Tensor scratch =
        at::empty({2 * stat + rows_n * parts * D * 2}, q.options().dtype(ScalarType::Byte));
    char* sp = static_cast<char*>(scratch.data_ptr());
    p.exp_sums = reinterpret_cast<float*>(sp);
    p.max_logits = reinterpret_cast<float*>(sp + stat);
    p.tmp_out = sp + 2 * stat;
    p.max_num_partitions = static_cast<int32_t>(parts);
    run(nullptr, true);
    return true;
  });
}

PyMethodDef kMethods[] = {
    {"paged_attention_v1", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_v1)), METH_FASTCALL, nullptr},
    {"paged_attention_v2", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_v2)), METH_FASTCALL, nullptr},
    {"reshape_and_cache", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_write_x)), METH_FASTCALL,
     nullptr},
    {"reshape_and_cache_flash", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_write_flash)),
     METH_FASTCALL, nullptr},
    {"attention_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_step)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_C_b200", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__C_b200() { return PyModule_Create(&kModule); }
