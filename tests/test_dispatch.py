"""The rules that pick a kernel for a call, asked on the host (no GPU: a chip of 148 SMs is assumed)."""
import subprocess
from pathlib import Path

import pytest

from vllm_b200 import capi


def _route(seqs, heads, kv_heads, head_size, max_len, kv=0, dtype=capi.BF16, block=16):
    a = capi.AttnArgs()
    a.num_seqs, a.num_heads, a.num_kv_heads, a.head_size = seqs, heads, kv_heads, head_size
    a.block_size, a.max_seq_len, a.kv_dtype, a.q_dtype = block, max_len, kv, dtype
    a.q_stride = heads * head_size
    a.kv_head_stride, a.kv_block_stride = head_size * block, kv_heads * head_size * block
    return capi.decode_route(a)


@pytest.mark.parametrize("seqs,max_len", [(1, 32000), (4, 32000), (1, 131072)])
def test_head_size_120_keeps_its_cluster_however_long_the_sequences_are(seqs, max_len):
    # only the direct kernel is built for it: as many CTAs as for sequences where it is the better one
    assert _route(seqs, 32, 8, 120, max_len) == _route(seqs, 32, 8, 120, 2048) > 1


def test_head_size_120_long_sequences_fill_one_wave():
    # 256 items: a cluster of 2 each would be 512 CTAs for 444 places
    assert _route(64, 4, 4, 120, 8000) == 1 and _route(32, 4, 4, 120, 8000) == 2


def test_head_sizes_with_both_kernels_leave_long_sequences_to_the_persistent_one():
    assert _route(1, 32, 8, 128, 32000) == 0
    assert _route(1, 32, 8, 128, 1500) > 1
    assert _route(1, 32, 8, 128, 1500, dtype=capi.F32) == -1


# (sequences, heads, kv heads, head size, longest, fp8 cache), where one of the two kernels took at least a
# sixth longer on a B200 with all sequences equally long.  (The rule leaves batches of several waves that it
# estimates at up to 1.15, or 1.25 with one small wave more, to the direct kernel, where spread lengths gain.)
@pytest.mark.parametrize("call", [(32, 8, 8, 128, 2500, 1), (256, 8, 8, 128, 200, 1), (32, 8, 8, 80, 2500, 1),
                                  (256, 32, 8, 80, 200, 1), (256, 64, 8, 96, 200, 1), (64, 32, 32, 96, 1000, 1), (256, 8, 8, 64, 200, 1),
                                  (32, 32, 8, 128, 2500, 0)])
def test_batches_that_the_persistent_kernel_serves_faster(call):
    assert _route(*call[:5], kv=call[5]) == 0


@pytest.mark.parametrize("call", [(1, 32, 8, 128, 1500, 0), (8, 32, 32, 128, 1024, 0), (8, 32, 8, 64, 300, 1),
                                  (16, 16, 1, 128, 2000, 0), (1, 8, 8, 32, 8000, 0), (64, 64, 4, 128, 300, 1),
                                  (4, 32, 8, 256, 1000, 1), (32, 64, 4, 112, 2500, 0), (12, 32, 8, 128, 3000, 0)])
def test_batches_that_the_direct_kernel_serves_faster(call):
    assert _route(*call[:5], kv=call[5]) > 0


def test_a_gpu_without_room_for_clusters_of_16_gets_smaller_ones(tmp_path):
    """The size is asked from the GPU; here from a stand-in that has room up to some size."""
    (tmp_path / "t.cpp").write_text("""
#include <cstdio>
#include "cluster_fit.h"
int main() {
  const int most[] = {16, 15, 8, 7, 4, 1, 0};
  for (int m : most) std::printf("%d ", b200pa::largest_cluster([&](int n) { return n <= m ? 132 / n : 0; }));
  std::printf("%d\\n", b200pa::largest_cluster([](int) { return -1; }));
}
""")
    csrc = Path(__file__).resolve().parents[1] / "vllm_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", f"-I{csrc}", "t.cpp", "-o", "t"], cwd=tmp_path, check=True, timeout=120)
    out = subprocess.run(["./t"], cwd=tmp_path, check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["16", "8", "8", "4", "4", "1", "1", "1"]


def test_the_choice_of_v1_and_v2_is_the_reference_s():
    from vllm_b200.paged_attn import PagedAttention
    for max_len in (0, 1, 511, 512, 513, 8191, 8192, 8193, 100000):
        for seqs, heads in ((1, 1), (1, 512), (1, 513), (16, 32), (17, 32), (256, 64)):
            partitions = (max_len + 511) // 512
            assert PagedAttention.use_v1(max_len, seqs, heads) == (
                max_len <= 8192 and (partitions == 1 or seqs * heads > 512))
    assert capi.lib().b200pa_stream_workspace_bytes() == 4 << 20
