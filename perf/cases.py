"""Performance cases of the paged-attention path, through its public entry points.

Three kinds of work, told apart by ``case["op"]``:

  step       one engine step of one layer: the backend builds its metadata from what the engine
             hands over and runs ``forward`` (KV write, then attention) on a batch of decode
             requests (one new token) and prefill chunks (many)
  attention  ``paged_attention_v1`` / ``_v2`` on a decode batch whose cache is already written
  write      ``reshape_and_cache`` / ``_flash``: new tokens into the cache, on their own

Lengths are quantiles of the distribution that a case names, so that the work of a case follows
from the case alone; the seed decides their order, the block tables and every value.
"""
from __future__ import annotations

import math
import statistics
import types

import numpy as np
import torch

from vllm_b200 import _custom_ops as ops
from vllm_b200.backend import (B200PagedAttentionBackend, B200PagedAttentionImpl,
                               B200PagedAttentionMetadataBuilder)
from vllm_b200.paged_attn import _PARTITION_SIZE

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _heads(heads, kv_heads, head_size, block_size, dtype="bf16", kv="auto", alibi=False):
    return {"heads": heads, "kv_heads": kv_heads, "head_size": head_size, "block_size": block_size,
            "dtype": dtype, "kv": kv, "alibi": alibi}


def _step(decodes, dec_lo, dec_hi, chunks, chunk_lo, chunk_hi, ctx_lo, ctx_hi, **heads):
    """`decodes` requests with one new token and contexts in [dec_lo, dec_hi]; `chunks` requests
    with [chunk_lo, chunk_hi] new tokens each behind [ctx_lo, ctx_hi] cached ones."""
    return {"op": "step", "decodes": decodes, "dec_lo": dec_lo, "dec_hi": dec_hi, "chunks": chunks,
            "chunk_lo": chunk_lo, "chunk_hi": chunk_hi, "ctx_lo": ctx_lo, "ctx_hi": ctx_hi, **heads}


def _attention(version, seqs, lens, lo, hi, **heads):
    return {"op": "attention", "version": version, "seqs": seqs, "lens": lens, "lo": lo, "hi": hi,
            **heads}


def _write(layout, runs, run_lo, run_hi, **heads):
    """`runs` sequences, [run_lo, run_hi] new tokens each at consecutive positions."""
    return {"op": "write", "layout": layout, "runs": runs, "run_lo": run_lo, "run_hi": run_hi, **heads}


def listed():
    gqa8b = _heads(32, 8, 128, 16)
    gqa70b_fp8 = _heads(64, 8, 128, 16, kv="fp8")
    return [
        # one interactive user: every launch and every line of host code shows
        {"name": "step_decode_1", **_step(1, 1500, 1500, 0, 0, 0, 0, 0, **gqa8b)},
        # long prompts in chunks, part of each already cached: a prefill-heavy step at an
        # 8 k-token budget
        {"name": "step_prefill", **_step(0, 0, 0, 4, 1536, 2560, 0, 4096, **gqa8b)},
        # the everyday step of a busy server: decodes with a prompt's chunk riding along, fp8 cache
        {"name": "step_mixed_fp8", **_step(60, 200, 4000, 3, 150, 700, 0, 1500, **gqa70b_fp8)},
        # small multi-head batch, short ragged contexts
        {"name": "v1_mha_8", **_attention("v1", 8, "uniform", 1, 1024, **_heads(32, 32, 128, 16))},
        # the headline: a full decode batch of an 8B-shape layer
        {"name": "v2_gqa_256", **_attention("v2", 256, "uniform", 512, 4096, **gqa8b)},
        # a 70B-shape layer with an fp8 cache, long contexts
        {"name": "v2_fp8_128", **_attention("v2", 128, "uniform", 8192, 8192, **gqa70b_fp8)},
        # long-context batch with a heavy tail: a few sequences hold most of the tokens
        {"name": "v2_skewed_64", **_attention("v2", 64, "lognormal", 16, 32768, **gqa8b)},
        # the largest: a serving batch of 2048 sequences, fp8, 32-token blocks
        {"name": "v2_serving_2048", **_attention("v2", 2048, "uniform", 1024, 8192,
                                                 **_heads(64, 8, 128, 32, kv="fp8"))},
        # the other option set: fp16, ALiBi, multi-head, a head size that is no power of two
        {"name": "v1_alibi_33", **_attention("v1", 33, "uniform", 100, 3000,
                                             **_heads(40, 40, 80, 32, dtype="fp16", alibi=True))},
        # KV write of a prefill step, quantising
        {"name": "write_prefill_fp8", **_write("x", 128, 128, 128, **gqa70b_fp8)},
        # KV write of a decode step: one token per sequence, each in a block of its own
        {"name": "write_decode_256", **_write("x", 256, 1, 1, **gqa70b_fp8)},
        # the flash layout, ragged prompts, unquantised
        {"name": "write_flash_ragged", **_write("NHD", 13, 30, 900, **gqa8b)},
    ]


# ------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_heads(rng, alibi_too=True):
    head_size = 128 if rng.random() < 0.5 else rng.choice([32, 64, 80, 96, 112, 120, 192, 256])
    heads, kv_heads = rng.choice([(32, 8), (64, 8), (32, 32), (40, 40), (8, 2), (32, 2), (16, 1),
                                  (12, 4), (8, 8), (28, 4)])
    kv = rng.choice(["auto", "auto", "fp8", "fp8", "fp8_e5m2"])
    if head_size == 120:  # not a multiple of the 16 elements that an fp8 cache keeps together
        kv = "auto"
    return _heads(heads, kv_heads, head_size, rng.choice([16, 16, 32]),
                  rng.choice(["bf16", "bf16", "fp16"]), kv, alibi_too and rng.random() < 0.15)


def _range(rng, lo, hi):
    """A range of lengths inside [lo, hi], both ends spread over the logarithm."""
    a, b = sorted((_log(rng, lo, hi), _log(rng, lo, hi)))
    return a, b


def draw(rng):
    op = rng.choice(["step", "step", "attention", "attention", "write"])
    while True:
        if op == "step":
            kind = rng.choice(["decode", "prefill", "mixed"])
            decodes = 0 if kind == "prefill" else _log(rng, 1, 400)
            chunks = 0 if kind == "decode" else _log(rng, 1, 24)
            dec = _range(rng, 16, 12000) if decodes else (0, 0)
            chunk = _range(rng, 16, 4096) if chunks else (0, 0)
            ctx = (0, rng.choice([0, _log(rng, 16, 8192)])) if chunks else (0, 0)
            c = _step(decodes, *dec, chunks, *chunk, *ctx, **_draw_heads(rng))
        elif op == "attention":
            lens = rng.choice(["uniform", "uniform", "lognormal"])
            lo, hi = _range(rng, 1, 32768)
            c = _attention(rng.choice(["v1", "v2"]), _log(rng, 1, 1024), lens, lo, hi, **_draw_heads(rng))
        else:
            runs, lo, hi = _log(rng, 1, 512), 1, 1
            if rng.random() < 0.6:
                lo, hi = _range(rng, 1, 4096)
            c = _write(rng.choice(["x", "x", "NHD", "HND"]), runs, lo, hi, **_draw_heads(rng, False))
        w = work(c)
        new_tokens = sum(_plan(c)[1])
        if w["bytes"] <= 4e9 and w["flops"] <= 6e11 and new_tokens <= 65536 and \
                (op != "step" or new_tokens <= 9000):
            return c


# ------------------------------------------------------------------ lengths and work
def _quantiles(n, lo, hi):
    return [int(lo + (hi - lo) * (i + 0.5) / n + 0.5) for i in range(n)]


def _plan(case):
    """(length, new tokens) of every sequence, in no particular order."""
    if case["op"] == "attention":
        n = case["seqs"]
        if case["lens"] == "uniform":
            return _quantiles(n, case["lo"], case["hi"]), [0] * n
        z = statistics.NormalDist()
        lens = [math.exp(8.5 + z.inv_cdf((i + 0.5) / n)) for i in range(n)]
        return [int(min(max(v, case["lo"]), case["hi"])) for v in lens], [0] * n
    if case["op"] == "write":
        new = _quantiles(case["runs"], case["run_lo"], case["run_hi"])
        return [37 * (i % 11) + t for i, t in enumerate(new)], new  # (most runs start inside a block)
    lens = _quantiles(case["decodes"], case["dec_lo"], case["dec_hi"])
    new = [1] * case["decodes"]
    n = case["chunks"]
    chunk = _quantiles(n, case["chunk_lo"], case["chunk_hi"])
    for i, ctx in enumerate(_quantiles(n, case["ctx_lo"], case["ctx_hi"])):
        t = chunk[(5 * i + 2) % n] if n % 5 else chunk[(7 * i + 2) % n]  # (contexts and chunks mixed)
        lens.append(ctx + t)
        new.append(t)
    return lens, new


def _sizes(case):
    return 2, (2 if case["kv"] == "auto" else 1)  # bytes of an input element, of a cache element


def work(case):
    """Bytes: every sequence's K and V read once, q read, out written, block tables and lengths;
    for new tokens k and v read and their cache entries written.  Flops: q.k and p.v over the
    tokens that each query attends to."""
    lens, new = _plan(case)
    es, ec = _sizes(case)
    D, H, HK = case["head_size"], case["heads"], case["kv_heads"]
    n = sum(new)
    written = n * HK * D * 2 * (es + ec) + 8 * n
    if case["op"] == "write":
        return {"bytes": written, "flops": 0}
    table = 4 * sum(-(-v // case["block_size"]) for v in lens) + 8 * len(lens)
    if case["op"] == "attention":
        queries, pairs, old = len(lens), sum(lens), sum(lens)
    else:
        queries = n
        pairs = sum(t * (v - t) + t * (t + 1) // 2 for v, t in zip(lens, new))
        old = sum(lens) - n  # (the step's own tokens come in as k and v)
    kv = old * HK * D * 2 * ec
    return {"bytes": kv + 2 * queries * H * D * es + table + written, "flops": 4 * H * D * pairs}


def tolerance(case):
    """KV writes are bytes.  Attention results and P are rounded to 16 bits and the order of the
    sums is the implementation's."""
    return "exact" if case["op"] == "write" else {"rel": 1e-2}


# ------------------------------------------------------------------ inputs
def _fp8_type(kv):
    return (torch.float8_e5m2, 57344.0) if kv == "fp8_e5m2" else (torch.float8_e4m3fn, 448.0)


def _fill_cache(flat, case, scale, gen):
    """N(0, 1) keys and values, as the cache holds them."""
    step = 1 << 28
    for a in range(0, flat.numel(), step):
        part = flat[a:a + step]
        if case["kv"] == "auto":
            part.normal_(generator=gen)
        else:
            t, top = _fp8_type(case["kv"])
            x = torch.empty(part.numel(), dtype=torch.float16, device=DEV).normal_(generator=gen)
            part.copy_(x.mul_(1.0 / scale).clamp_(-top, top).to(t).view(torch.uint8))


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    lens, new = (np.array(v, dtype=np.int64) for v in _plan(case))
    order = rng.permutation(len(lens))
    if case["op"] == "step":  # the engine keeps its decode requests in front
        order = np.concatenate([order[new[order] == 1], order[new[order] != 1]])
    lens, new = lens[order], new[order]
    n, S = int(new.sum()), len(lens)
    D, H, HK, B = case["head_size"], case["heads"], case["kv_heads"], case["block_size"]
    dtype, fp8 = DTYPES[case["dtype"]], case["kv"] != "auto"
    cache_dtype = torch.uint8 if fp8 else dtype

    # blocks: one random permutation of a pool with a quarter to spare, dealt out
    need = np.maximum(1, -(-lens // B))
    nb = int(1.25 * need.sum()) + 8
    perm = rng.permutation(nb).astype(np.int32)
    start = np.concatenate([[0], np.cumsum(need)])
    table = np.zeros((S, int(need.max())), dtype=np.int32)
    for s in range(S):
        table[s, :need[s]] = perm[start[s]:start[s + 1]]
    seq = np.repeat(np.arange(S), new)
    pos = np.concatenate([np.arange(v - t, v) for v, t in zip(lens, new)]) if n else np.zeros(0, np.int64)
    slots = table[seq, pos // B].astype(np.int64) * B + pos % B

    # a per-tensor scale as calibration gives it: the largest magnitude onto the largest code
    scale = 5.3 / _fp8_type(case["kv"])[1] if fp8 else 1.0
    s = types.SimpleNamespace(case=case, kv=case["kv"], D=D, H=H, HK=HK, B=B, scale=D ** -0.5,
                              max_len=int(lens.max()))
    s.k_scale = torch.tensor(scale, dtype=torch.float32, device=DEV)
    s.v_scale = torch.tensor(scale, dtype=torch.float32, device=DEV)
    s.table = torch.from_numpy(table).to(DEV)
    s.lens = torch.from_numpy(lens.astype(np.int32)).to(DEV)
    s.slots = torch.from_numpy(slots).to(DEV)
    if n:
        s.key = torch.empty((n, HK, D), dtype=dtype, device=DEV).normal_(generator=gen)
        s.value = torch.empty((n, HK, D), dtype=dtype, device=DEV).normal_(generator=gen)
    slopes = [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)] if case["alibi"] else None

    if case["op"] == "write" and case["layout"] != "x":
        shape = (nb, B, HK, D) if case["layout"] == "NHD" else (nb, HK, B, D)
        caches = [torch.zeros(shape, dtype=cache_dtype, device=DEV) for _ in range(2)]
        s.key_cache, s.value_cache = caches if case["layout"] == "NHD" else [c.transpose(1, 2) for c in caches]
        return s
    if case["op"] == "step":
        shape = B200PagedAttentionBackend.get_kv_cache_shape(nb, B, HK, D, case["kv"])
        s.kv_cache = torch.empty(shape, dtype=cache_dtype, device=DEV)
        _fill_cache(s.kv_cache.view(-1), case, scale, gen)
        s.query = torch.empty((n, H, D), dtype=dtype, device=DEV).normal_(generator=gen)
        s.out = torch.empty((n, H * D), dtype=dtype, device=DEV)
        s.impl = B200PagedAttentionImpl(H, D, s.scale, HK, alibi_slopes=slopes, kv_cache_dtype=case["kv"])
        s.builder = B200PagedAttentionMetadataBuilder(types.SimpleNamespace(block_size=B), ["layer.0"],
                                                      None, torch.device(DEV))
        s.layer = types.SimpleNamespace(_k_scale=s.k_scale, _v_scale=s.v_scale)
        qsl = torch.from_numpy(np.concatenate([[0], np.cumsum(new)]).astype(np.int32))
        lens_cpu = torch.from_numpy(lens.astype(np.int32))
        s.common = types.SimpleNamespace(
            query_start_loc=qsl.to(DEV), query_start_loc_cpu=qsl, seq_lens=s.lens, seq_lens_cpu=lens_cpu,
            num_computed_tokens_cpu=torch.from_numpy((lens - new).astype(np.int32)), num_reqs=S,
            num_actual_tokens=n, max_query_len=int(new.max()), max_seq_len=s.max_len,
            block_table_tensor=s.table, slot_mapping=s.slots, causal=True)
        return s
    x = 16 // (1 if fp8 else 2)
    s.key_cache = torch.empty((nb, HK, D // x, B, x), dtype=cache_dtype, device=DEV)
    s.value_cache = torch.empty((nb, HK, D, B), dtype=cache_dtype, device=DEV)
    if case["op"] == "write":
        s.key_cache.zero_()
        s.value_cache.zero_()
        return s
    _fill_cache(s.key_cache.view(-1), case, scale, gen)
    _fill_cache(s.value_cache.view(-1), case, scale, gen)
    s.query = torch.empty((S, H, D), dtype=dtype, device=DEV).normal_(generator=gen)
    s.alibi = torch.tensor(slopes, dtype=torch.float32, device=DEV) if slopes else None
    s.out = torch.empty_like(s.query)
    if case["version"] == "v2":
        parts = -(-s.max_len // _PARTITION_SIZE)
        s.exp_sums = torch.empty((S, H, parts), dtype=torch.float32, device=DEV)
        s.max_logits = torch.empty_like(s.exp_sums)
        s.tmp_out = torch.empty((S, H, parts, D), dtype=dtype, device=DEV)
    return s


def run(s):
    op = s.case["op"]
    if op == "step":
        metadata = s.builder.build(0, s.common)
        s.impl.forward(s.layer, s.query, s.key, s.value, s.kv_cache, metadata, output=s.out)
        return {"out": s.out, "kv_cache": s.kv_cache}
    if op == "attention":
        if s.case["version"] == "v1":
            ops.paged_attention_v1(s.out, s.query, s.key_cache, s.value_cache, s.HK, s.scale, s.table,
                                   s.lens, s.B, s.max_len, s.alibi, s.kv, s.k_scale, s.v_scale)
        else:
            ops.paged_attention_v2(s.out, s.exp_sums, s.max_logits, s.tmp_out, s.query, s.key_cache,
                                   s.value_cache, s.HK, s.scale, s.table, s.lens, s.B, s.max_len,
                                   s.alibi, s.kv, s.k_scale, s.v_scale)
        return s.out
    write = ops.reshape_and_cache if s.case["layout"] == "x" else ops.reshape_and_cache_flash
    write(s.key, s.value, s.key_cache, s.value_cache, s.slots, s.kv, s.k_scale, s.v_scale)
    return {"key_cache": s.key_cache, "value_cache": s.value_cache}
