"""The direct decode kernel (small batches: one cluster per (sequence, kv head)) at the sizes where its
tiling can go wrong, and the persistent kernel on the parity tests that small batches no longer
send to it."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

from test_attention_gpu import DEV, check
from vllm_b200 import _custom_ops as ops
import workloads as W

pytestmark = pytest.mark.gpu


def _workload(lens, hq, hkv, d, block, dtype, kv, seed=5):
    lens = np.array(lens)
    w = W.make_decode("direct", num_seqs=len(lens), num_heads=hq, num_kv_heads=hkv, head_size=d,
                      block_size=block, lens=lens, dtype=dtype, kv_cache_dtype=kv, device=DEV, seed=seed,
                      rng=np.random.default_rng(seed))
    w.query.mul_(6.0)
    return w


# clusters of 1 (max length 64) to 16 (length 2048 and more, eight items at most); tiles of 16 tokens
@pytest.mark.parametrize("lens", [[0, 1], [1, 15, 16, 17], [63, 64, 65], [127, 128, 129, 0], [511, 513],
                                  [2047], [2049, 3]])
@pytest.mark.parametrize("heads", [(8, 1), (9, 1), (4, 4)])
@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_tile_and_cluster_edges(lens, heads, kv):
    for block in (16, 32):
        check(_workload(lens, *heads, 128, block, torch.bfloat16, kv), "v1")


@pytest.mark.parametrize("d", [32, 64, 80, 96, 112, 120, 128, 192, 256])
@pytest.mark.parametrize("kv,dtype", [("auto", torch.float16), ("fp8_e5m2", torch.bfloat16)])
def test_head_sizes(d, kv, dtype):
    if d == 120 and kv != "auto":
        pytest.skip("an fp8 cache keeps 16 head dimensions together")
    for heads in ((6, 2), (24, 2)):
        check(_workload([700, 33, 1], *heads, d, 16, dtype, kv), "v2")


def test_head_size_120_large_batch():
    check(_workload(np.random.default_rng(0).integers(1, 600, size=200), 4, 4, 120, 16, torch.bfloat16, "auto"),
          "v1", seqs=range(0, 200, 17))


@pytest.mark.parametrize("lens", [[32000], [20000, 31999, 7, 513]])
def test_head_size_120_long_sequences(lens):
    for heads in ((8, 2), (24, 2)):
        check(_workload(lens, *heads, 120, 16, torch.bfloat16, "auto"), "v2")


def test_lse_and_stale_nans():
    w = _workload([129, 40], 8, 2, 128, 16, torch.bfloat16, "auto")
    for s, n in enumerate((129, 40)):
        blk = w.block_tables[s, n // 16].long()
        w.key_cache[blk, :, :, n % 16:] = float("nan")
        w.value_cache[blk, :, :, n % 16:] = float("nan")
    out, lse = torch.empty_like(w.query), torch.empty((8, 2), dtype=torch.float32, device=DEV)
    ops.paged_attention_with_lse(out, lse, w.query, w.key_cache, w.value_cache, 2, w.scale, w.block_tables,
                                 w.seq_lens, 16, w.max_seq_len, None, "auto", w.k_scale, w.v_scale)
    for s, n in enumerate((129, 40)):
        blocks = w.block_tables[s, :(n + 15) // 16].long()
        k = w.key_cache[blocks].permute(1, 0, 3, 2, 4).reshape(2, -1, 128)[:, :n].float()
        logits = torch.einsum("hgd,hld->hgl", w.query[s].float().view(2, 4, 128), k) * w.scale
        torch.testing.assert_close(lse[:, s], logits.logsumexp(-1).view(8), atol=1e-3, rtol=1e-3)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("direct", ["1", "2"], ids=["direct", "persistent"])
def test_both_decode_kernels_pass_the_parity_tests(direct):
    """B200PA_TUNE_DIRECT forces one kernel for every call it is built for (read once per process)."""
    root = Path(__file__).resolve().parents[1]
    files = [str(root / "tests" / f) for f in ("test_attention_gpu.py", "test_lse_gpu.py")]
    r = subprocess.run(
        [sys.executable, "-m", "pytest", *files, "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"],
        env=dict(os.environ, B200PA_TUNE_DIRECT=direct), cwd=str(root), capture_output=True, text=True,
        timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
