"""Whole engine steps through the backend (KV write and attention in one call) at the places where a
step is divided between kernels: captured steps replayed with other batches, decodes beside chunks on
either stream, the native step against the operators one by one."""
import types

import numpy as np
import pytest
import torch

from test_prefill_gpu import _gather
from vllm_b200.backend import (B200PagedAttentionBackend, B200PagedAttentionImpl,
                               B200PagedAttentionMetadataBuilder)

pytestmark = pytest.mark.gpu
DEV = "cuda"


class Engine:
    """Static buffers for up to `reqs` requests and `tokens` tokens, and a cache full of old tokens."""

    def __init__(self, reqs, tokens, H=8, HK=2, D=128, B=16, max_blocks=40, kv="auto", alibi=False, seed=0):
        self.H, self.HK, self.D, self.B, self.kv = H, HK, D, B, kv
        self.rng = np.random.default_rng(seed)
        self.gen = torch.Generator(device=DEV).manual_seed(seed)
        self.dtype = torch.bfloat16
        self.scale = 0.02 if kv != "auto" else 1.0
        self.nb = reqs * max_blocks + 1
        shape = B200PagedAttentionBackend.get_kv_cache_shape(self.nb, B, HK, D, kv)
        old = torch.randn(shape, generator=self.gen, device=DEV)
        if kv == "auto":
            self.cache = old.to(self.dtype)
        else:
            t = torch.float8_e5m2 if kv == "fp8_e5m2" else torch.float8_e4m3fn
            self.cache = (old / self.scale).clamp(-448, 448).to(t).view(torch.uint8)
        del old
        self.q, self.k, self.v = (self._randn(tokens, h, D) for h in (H, HK, HK))
        self.out = torch.zeros(tokens, H * D, dtype=self.dtype, device=DEV)
        self.qsl = torch.zeros(reqs + 1, dtype=torch.int32, device=DEV)
        self.lens = torch.zeros(reqs, dtype=torch.int32, device=DEV)
        self.table = torch.zeros(reqs, max_blocks, dtype=torch.int32, device=DEV)
        self.slots = torch.full((tokens,), -1, dtype=torch.int64, device=DEV)
        slopes = [2.0 ** (-(i + 1) / 2) for i in range(H)] if alibi else None
        self.impl = B200PagedAttentionImpl(H, D, D ** -0.5, HK, alibi_slopes=slopes, kv_cache_dtype=kv)
        self.builder = B200PagedAttentionMetadataBuilder(types.SimpleNamespace(block_size=B), ["l"], None, DEV)
        scale = torch.tensor(self.scale, dtype=torch.float32, device=DEV)
        self.layer = types.SimpleNamespace(_k_scale=scale, _v_scale=scale)

    def _randn(self, *shape):
        return torch.randn(*shape, generator=self.gen, device=DEV).to(self.dtype)

    def load(self, new, ctx):
        """Fills the buffers with a batch; the requests behind it bring no token."""
        self.new, self.ctx = np.array(new), np.array(ctx)
        n, r = int(self.new.sum()), len(new)
        for t in (self.q, self.k, self.v):
            t.copy_(self._randn(*t.shape))
        table = self.rng.permutation(self.nb - 1)[: self.table.numel()].reshape(self.table.shape) + 1
        self.table.copy_(torch.from_numpy(table.astype(np.int32)))
        offsets = np.full(self.qsl.numel(), n, np.int32)
        offsets[: r + 1] = np.concatenate([[0], np.cumsum(self.new)])
        lens = np.zeros(self.lens.numel(), np.int32)
        lens[:r] = self.new + self.ctx
        slots = np.full(self.slots.numel(), -1, np.int64)
        seq = np.repeat(np.arange(r), self.new)
        pos = np.concatenate([np.arange(c, c + t) for t, c in zip(new, ctx)])
        slots[:n] = table[seq, pos // self.B] * self.B + pos % self.B
        self.qsl.copy_(torch.from_numpy(offsets))
        self.lens.copy_(torch.from_numpy(lens))
        self.slots.copy_(torch.from_numpy(slots))
        self.out.fill_(float("nan"))

    def common(self, max_query_len=None, max_seq_len=None, tokens=None):
        qsl = self.qsl.cpu()
        return types.SimpleNamespace(
            query_start_loc=self.qsl, query_start_loc_cpu=qsl, seq_lens=self.lens, seq_lens_cpu=self.lens.cpu(),
            num_reqs=self.lens.numel(), num_actual_tokens=tokens or int(qsl[-1]),
            max_query_len=max_query_len or int(qsl.diff().max()),
            max_seq_len=max_seq_len or int(self.lens.max()), block_table_tensor=self.table,
            slot_mapping=self.slots, causal=True)

    def forward(self, metadata):
        self.impl.forward(self.layer, self.q, self.k, self.v, self.cache, metadata, output=self.out)

    def check(self):
        """The rows of the loaded batch against dense attention in fp32 over what the cache holds."""
        torch.cuda.synchronize()
        H, HK, D, g = self.H, self.HK, self.D, self.H // self.HK
        x = 16 // self.cache.element_size()
        kc = self.cache[0].view(self.nb, HK, D // x, self.B, x)
        vc = self.cache[1].view(self.nb, HK, D, self.B)
        slopes = self.impl.alibi_slopes
        off = 0
        for r, (t, c) in enumerate(zip(self.new, self.ctx)):
            if t == 0:
                continue
            k, v = _gather(kc, vc, self.table[r], int(t + c), self.kv, self.scale)
            if self.kv == "auto":
                assert torch.equal(k[c:], self.k[off:off + t].float())
            qq = self.q[off:off + t].float().view(t, HK, g, D)
            s = torch.einsum("tkgd,lkd->kgtl", qq, k) * D ** -0.5
            pos, key = torch.arange(c, c + t, device=DEV).view(-1, 1), torch.arange(c + t, device=DEV).view(1, -1)
            if slopes is not None:
                s = s + slopes.to(DEV).view(HK, g, 1, 1) * (key - pos).float()
            s = s.masked_fill(key > pos, float("-inf"))
            want = torch.einsum("kgtl,lkd->tkgd", torch.softmax(s, -1), v).reshape(t, H * D)
            got = self.out[off:off + t].float()
            # (P and the result are rounded to 16 bits: 2^-9 each, and 2^-9 of partials that were cut)
            assert (got - want).norm() < 6e-3 * want.norm(), (r, t, c)
            torch.testing.assert_close(got, want, atol=2e-2, rtol=2e-2)
            off += t
        from vllm_b200 import capi
        assert capi.device_status() == 0


def _capture(e, metadata):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        e.forward(metadata)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        e.forward(metadata)
    return g


@pytest.mark.parametrize("kv", ["auto", "fp8"])
@pytest.mark.parametrize("for_capture", [True, False], ids=["build_for_cudagraph_capture", "build"])
def test_a_captured_step_is_replayed_with_other_divisions_of_its_tokens(kv, for_capture):
    e = Engine(8, 8, kv=kv)
    e.load([1] * 8, [20 * i for i in range(8)])
    common = e.common(max_query_len=8, max_seq_len=640)  # as an engine's dummy run has it
    g = _capture(e, e.builder.build_for_cudagraph_capture(common) if for_capture else e.builder.build(0, common))
    for new, ctx in (([1, 1, 4, 1, 1], [300, 5, 77, 0, 500]), ([8], [600]), ([1] * 8, [40 * i for i in range(8)]),
                     ([3, 1, 1, 1, 2], [0, 17, 128, 255, 31]), ([1, 0, 7], [9, 0, 3])):
        e.load(new, ctx)
        g.replay()
        e.check()


def test_a_step_without_a_prefill_kernel_writes_its_kv_once():
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import capi
    e = Engine(4, 32, B=8)  # (block size 8: decode kernels only)
    e.load([1, 1, 20, 7], [30, 100, 50, 0])
    md = e.builder.build(0, e.common())

    def launches(f):
        capi.launch_count(reset=True)
        f()
        return capi.launch_count()
    step = launches(lambda: e.forward(md))
    e.check()
    kc, vc = e.cache[0].view(e.nb, e.HK, e.D // 8, 8, 8), e.cache[1].view(e.nb, e.HK, e.D, 8)
    write = launches(lambda: ops.reshape_and_cache(e.k, e.v, kc, vc, e.slots, "auto", e.layer._k_scale,
                                                   e.layer._v_scale))
    e.impl.kv_sharing_target_layer_name = "another layer writes"
    assert step == launches(lambda: e.forward(md)) + write


@pytest.mark.parametrize("kv", ["auto", "fp8"])
@pytest.mark.parametrize("stream", ["first", "second"])
def test_split_decodes_and_cut_chunks_share_the_workspace(stream, kv):
    """Long decodes go to the persistent kernel, split across warps through one half of the stream's
    workspace, while the prefill kernel runs beside it on the other half."""
    from vllm_b200 import capi
    e = Engine(6, 400, max_blocks=2000, kv=kv)
    a = capi.AttnArgs()
    a.num_seqs, a.num_heads, a.num_kv_heads, a.head_size, a.block_size = 3, e.H, e.HK, e.D, e.B
    a.max_seq_len, a.q_dtype, a.kv_dtype = 31000, capi.BF16, 0 if kv == "auto" else 1
    assert capi.decode_route(a) == 0
    with torch.cuda.stream(torch.cuda.current_stream() if stream == "first" else torch.cuda.Stream()):
        for _ in range(3):
            e.load([1, 1, 1, 20, 300, 9], [30999, 20000, 7, 25000, 2000, 9000])
            e.forward(e.builder.build(0, e.common()))
            e.check()


@pytest.mark.parametrize("new,ctx", [([1, 1, 1], [0, 700, 33]), ([1, 1, 9, 40], [300, 5, 0, 77]),
                                     ([5, 64], [0, 129]), ([1], [1500])])
@pytest.mark.parametrize("D,kv,alibi", [(128, "auto", False), (128, "fp8", True), (64, "fp8_e5m2", False),
                                        (120, "auto", True), (256, "auto", False)])
def test_the_native_step_does_what_the_operators_do(new, ctx, D, kv, alibi, monkeypatch):
    from vllm_b200 import _custom_ops as ops
    e = Engine(4, 80, D=D, kv=kv, alibi=alibi, max_blocks=100)
    # rows of a fused projection: strided by token
    fused = torch.empty(80, (e.H + 2 * e.HK) * D, dtype=e.dtype, device=DEV)
    e.q, e.k, e.v = (t.view(80, -1, D) for t in fused.split([e.H * D, e.HK * D, e.HK * D], dim=1))
    e.load(new, ctx)
    before = e.cache.clone()
    md = e.builder.build(0, e.common())
    step, taken = ops.attention_step, []
    monkeypatch.setattr(ops, "attention_step", lambda *args: taken.append(step(*args)) or taken[-1])
    e.forward(md)
    assert taken == [True]
    e.check()
    native, written = e.out.clone(), e.cache.clone()
    e.cache.copy_(before)
    e.out.fill_(float("nan"))
    monkeypatch.setattr(ops, "attention_step", lambda *args: False)
    e.forward(md)
    e.check()
    assert torch.equal(e.cache, written)
    n = sum(new)
    # (the same roundings in another order: two results of 16 bits, and partials of 16 bits in one of them)
    assert (e.out[:n].float() - native[:n].float()).norm() < 6e-3 * native[:n].float().norm()
    assert e.out[n:].isnan().all() and native[n:].isnan().all()


@pytest.mark.parametrize("new,ctx,scratch", [([1, 1, 1], [0, 700, 33], False), ([1] * 3, [9000, 20, 5000], True),
                                             ([1, 1, 9, 40], [300, 5, 0, 77], False), ([5, 64], [0, 129], False)])
@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_the_step_of_the_c_interface(new, ctx, scratch, kv):
    """b200pa_attention_step against the write and the attention as two calls, and without a write."""
    from vllm_b200 import capi
    e = Engine(len(new), sum(new), kv=kv, max_blocks=600)
    e.load(new, ctx)
    n, r = sum(new), len(new)
    chunks, decodes = max(new) > 1, new.count(1)
    x = 16 // e.cache.element_size()
    a = capi.AttnArgs(out=e.out.data_ptr(), query=e.q.data_ptr(), key_cache=e.cache[0].data_ptr(),
                      value_cache=e.cache[1].data_ptr(), block_tables=e.table.data_ptr(), seq_lens=e.lens.data_ptr(),
                      k_scale=e.layer._k_scale.data_ptr(), v_scale=e.layer._v_scale.data_ptr(), q_stride=e.H * e.D,
                      kv_block_stride=e.HK * e.D * e.B, kv_head_stride=e.D * e.B, num_seqs=r, num_heads=e.H,
                      num_kv_heads=e.HK, head_size=e.D, block_size=e.B, max_seq_len=int(e.lens.max()),
                      max_num_blocks_per_seq=e.table.shape[1], scale=e.D ** -0.5, q_dtype=capi.BF16,
                      kv_dtype=capi.kv_dtype_from_string(kv))
    if scratch:
        parts = a.max_num_partitions = -(-a.max_seq_len // 512)
        sums, tops = (torch.empty(r, e.H, parts, device=DEV) for _ in range(2))
        tmp = torch.empty(r, e.H, parts, e.D, dtype=e.dtype, device=DEV)
        a.exp_sums, a.max_logits, a.tmp_out = sums.data_ptr(), tops.data_ptr(), tmp.data_ptr()
    w = capi.CacheArgs(key=e.k.data_ptr(), value=e.v.data_ptr(), key_cache=a.key_cache, value_cache=a.value_cache,
                       slot_mapping=e.slots.data_ptr(), k_scale=a.k_scale, v_scale=a.v_scale, key_stride=e.HK * e.D,
                       value_stride=e.HK * e.D, num_tokens=n, num_heads=e.HK, head_size=e.D, block_size=e.B, x=x,
                       in_dtype=capi.BF16, kv_dtype=a.kv_dtype)
    before, starts = e.cache.clone(), e.qsl.data_ptr() if chunks else 0
    st = torch.cuda.current_stream().cuda_stream
    capi.attention_step(w, a, starts, n, decodes, scratch, st)
    e.check()
    got, written = e.out.clone(), e.cache.clone()
    e.cache.copy_(before)
    e.out.fill_(float("nan"))
    capi.reshape_and_cache(w, st)
    assert torch.equal(e.cache, written)
    capi.attention_step(None, a, starts, n, decodes, scratch, st)
    e.check()
    # (the same kernels on the same values: only the order of partial sums may differ)
    assert (got.float() - e.out.float()).norm() < 4e-3 * got.float().norm()

    # no kernel for the chunks: nothing is launched, the write neither
    if chunks:
        w.block_size = a.block_size = 8
        e.cache.copy_(before)
        capi.launch_count(reset=True)
        with pytest.raises(RuntimeError, match="no kernel"):
            capi.attention_step(w, a, starts, n, decodes, scratch, st)
        assert capi.launch_count() == 0 and torch.equal(e.cache, before)


def test_a_replay_beside_launches_on_another_stream():
    """A captured launch does not share its work-distribution words with ordinary ones: more of them
    than there are rotating slots run beside the replays."""
    graphed, eager = Engine(4, 512, max_blocks=60, seed=1), Engine(4, 512, max_blocks=60, seed=2)
    graphed.load([200, 100, 150, 62], [300, 7, 0, 500])
    eager.load([90, 128, 200, 30], [600, 70, 1, 250])
    g = _capture(graphed, graphed.builder.build(0, graphed.common()))
    md = eager.builder.build(0, eager.common())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(10):
        graphed.out.fill_(float("nan"))
        for _ in range(30):
            g.replay()
            with torch.cuda.stream(side):
                eager.forward(md)
        torch.cuda.current_stream().wait_stream(side)
        side.wait_stream(torch.cuda.current_stream())
    graphed.check()
    eager.check()


@pytest.mark.parametrize("kv", ["auto", "fp8"])
@pytest.mark.parametrize("new,ctx", [([1] * 3, [300, 15, 600]), ([1] * 120, list(range(60, 300, 2))),
                                     ([40, 130, 7], [100, 0, 500]), ([1] * 9 + [70, 33], [200] * 9 + [64, 300]),
                                     ([1500, 1400, 1300], [100, 0, 37])],  # (the write goes by tiles)
                         ids=["few-decodes", "many-decodes", "chunks", "mixed", "large-chunks"])
def test_attention_starts_under_the_write_of_its_step(new, ctx, kv):
    """Attention reads lengths, block tables and Q while the KV write in front may still run: what kernels
    before the write have just stored has to be what it sees, step after step, without a host in between."""
    eng = Engine(len(new), sum(new), kv=kv, max_blocks=max(40, -(-(max(new) + max(ctx)) // 16)))
    cache, names = eng.cache.clone(), ("q", "k", "v", "table", "lens", "slots", "qsl")
    steps = []
    for i in range(4):
        eng.load(new, [max(0, c - 7 * i) for c in ctx])
        steps.append({n: getattr(eng, n).clone() for n in names})
    meta = eng.builder.build(0, eng.common(max_seq_len=max(c + t for t, c in zip(new, ctx))))

    def run(wait):
        eng.cache.copy_(cache)
        outs = []
        for step in steps * 5:
            for n in names:
                getattr(eng, n).copy_(step[n])
            wait()
            eng.forward(meta)
            wait()
            outs.append(eng.out.clone())
        return torch.stack(outs).float()
    got, want = run(lambda: None), run(torch.cuda.synchronize)
    # (the same kernels on the same values: only the order of partial sums may differ)
    assert ((got - want).norm(dim=-1) < 4e-3 * want.norm(dim=-1)).all()
    from vllm_b200 import capi
    assert capi.device_status() == 0


@pytest.mark.parametrize("kv", ["auto", "fp8"])
@pytest.mark.parametrize("new,ctx", [([1] * 3, [300, 15, 600]), ([1] * 3, [9000, 20, 5000]), ([1] * 90, list(range(90, 180))),
                                     ([40, 130, 7], [100, 0, 500]), ([20, 9], [9000, 4000]),
                                     ([1, 1, 1, 20, 300], [9000, 700, 7, 8000, 500]), ([1500, 1400, 1300], [100, 0, 37])],
                         ids=["few-decodes", "split-decodes", "many-decodes", "chunks", "cut-chunks", "mixed", "large-chunks"])
def test_layers_back_to_back(new, ctx, kv):
    """Layers with caches of their own on one stream and no other kernel between: the result of a layer is the query
    of the next, so an attention kernel that read Q before the write in front of it has waited for the layer before,
    or met scheduler words, counters or partials of that layer's launches, would give other values.  Again with the
    next step's tokens, lengths and tables."""
    e = Engine(len(new), sum(new), kv=kv, max_blocks=max(50, -(-(max(new) + max(ctx) + 1) // 16)))
    n = 5
    bufs = [{"q": e.q, "k": e.k.clone(), "v": e.v.clone(), "out": e.out.clone(), "cache": e.cache.clone()}
            for _ in range(n)]
    for a, b in zip(bufs, bufs[1:]):
        b["q"] = a["out"].view(e.q.shape)

    def layer(b):
        for name, t in b.items():
            setattr(e, name, t)
    for step in range(3):
        layer({"q": bufs[0]["q"], "k": bufs[0]["k"], "v": bufs[0]["v"], "out": bufs[0]["out"]})
        e.load(new, [max(0, c - 7 * step) for c in ctx])
        for b in bufs:
            for name in ("k", "v", "out"):
                b[name].copy_(e._randn(*b[name].shape))
        meta = e.builder.build(0, e.common())
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)  # (all launches are there before the first one runs)
        for b in bufs:
            layer(b)
            e.forward(meta)
        for b in bufs:
            layer(b)
            e.check()
