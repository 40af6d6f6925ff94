"""Attention of steps whose requests bring several query tokens (paged_attention_varlen), against
fp32 dense causal attention over the same cache contents."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gather(key_cache, value_cache, table, n, kv, scale):
    """K and V [n, Hkv, D] of one request's first n positions, as fp32."""
    def plain(t):
        if kv == "auto":
            return t.float()
        return t.view(torch.float8_e5m2 if kv == "fp8_e5m2" else torch.float8_e4m3fn).float() * scale
    nb, hk, dx, B, x = key_cache.shape
    blocks = table[: (n + B - 1) // B].long()
    k = plain(key_cache[blocks]).permute(0, 3, 1, 2, 4).reshape(-1, hk, dx * x)[:n]
    v = plain(value_cache[blocks]).permute(0, 3, 1, 2).reshape(-1, hk, dx * x)[:n]
    return k, v


def _case(q_lens, ctx, H, HK, D, B, dtype, kv, alibi=False, seed=0, poison=True, ramp=0.0, dark=None):
    from vllm_b200 import _custom_ops as ops
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.default_rng(seed)
    q_lens, ctx = np.asarray(q_lens), np.asarray(ctx)
    lens = q_lens + ctx
    need = np.maximum(1, -(-lens // B))
    nb = int(need.sum()) + 3
    perm = rng.permutation(nb).astype(np.int32)
    table = np.zeros((len(lens), int(need.max())), np.int32)
    off = 0
    for r, k in enumerate(need):
        table[r, :k] = perm[off:off + k]
        off += k
    table = torch.from_numpy(table).to(DEV)
    fp8 = kv != "auto"
    x = 16 if fp8 else 16 // torch.empty((), dtype=dtype).element_size()
    scale = 0.02 if fp8 else 1.0
    kf = torch.randn((nb, HK, D // x, B, x), generator=gen, device=DEV)
    vf = torch.randn((nb, HK, D, B), generator=gen, device=DEV)
    for r, k in enumerate(need):  # logits that grow along the sequence
        kf[table[r, :k].long()] *= 1 + ramp * torch.arange(int(k), device=DEV).view(-1, 1, 1, 1, 1)
    if fp8:
        t = torch.float8_e5m2 if kv == "fp8_e5m2" else torch.float8_e4m3fn
        kc, vc = ((f / scale).clamp(-448, 448).to(t).view(torch.uint8) for f in (kf, vf))
    else:
        kc, vc = kf.to(dtype), vf.to(dtype)
    n = int(q_lens.sum())
    q = (2 * torch.randn((n, H, D), generator=gen, device=DEV)).to(dtype)
    out = torch.full((n, H, D), float("nan"), dtype=dtype, device=DEV)
    slopes = torch.tensor([2.0 ** (-(i + 1) / 2) for i in range(H)], device=DEV) if alibi else None
    if dark is not None:  # keys whose logits are -inf; those of the others lie around `low`
        first, low = dark
        q[..., 0] = q[..., 0].abs() + 0.5
        q[..., 1] = 4.0
        for r, n_keys in enumerate(lens):
            key = torch.arange(int(need[r]) * B, device=DEV)
            hidden = ((key < first) | (key % 128 >= 20)) & (key < int(ctx[r]))
            blocks = kc[table[r, :need[r]].long()].view(dtype if kv == "auto" else torch.float8_e5m2)
            k0 = blocks[:, :, 0, :, 0].float()
            k0.masked_fill_(hidden.view(-1, 1, B), float("-inf"))
            blocks[:, :, 0, :, 0] = k0.to(blocks.dtype)
            blocks[:, :, 0, :, 1] = torch.tensor(low / (4.0 * D ** -0.5 * scale)).to(blocks.dtype)
            kc[table[r, :need[r]].long()] = blocks.view(kc.dtype)
    if poison:  # stale bytes behind the end of a sequence must not reach the result
        bad = 0x7F if fp8 else float("nan")
        for r, k in enumerate(lens):
            if k % B:
                blk = table[r, k // B].long()
                kc[blk, :, :, k % B:] = bad
                vc[blk, :, :, k % B:] = bad
    qsl = torch.from_numpy(np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)).to(DEV)
    lens_t = torch.from_numpy(lens.astype(np.int32)).to(DEV)
    nd = int(np.argmax(q_lens != 1)) if (q_lens != 1).any() else len(q_lens)
    ks = torch.tensor(scale, device=DEV)
    took = ops.paged_attention_varlen(out, q, kc, vc, HK, D ** -0.5, table, lens_t, qsl, nd, B,
                                      int(lens.max()), slopes, kv, ks, ks)
    assert took
    torch.cuda.synchronize()
    off = 0
    for r, (t, c) in enumerate(zip(q_lens, ctx)):
        if t == 0:
            continue
        k, v = _gather(kc, vc, table[r], int(t + c), kv, scale)
        g = H // HK
        qq = q[off:off + t].float().view(t, HK, g, D)
        s = torch.einsum("tkgd,lkd->kgtl", qq, k) * D ** -0.5
        pos = torch.arange(c, c + t, device=DEV)
        key = torch.arange(c + t, device=DEV)
        if alibi:
            s = s + slopes.view(HK, g, 1, 1) * (key.view(1, -1) - pos.view(-1, 1)).float()
        s = s.masked_fill(key.view(1, -1) > pos.view(-1, 1), float("-inf"))
        want = torch.einsum("kgtl,lkd->tkgd", torch.softmax(s, -1), v).reshape(t, H, D)
        got = out[off:off + t].float()
        err = (got - want).norm() / want.norm()
        assert err < 6e-3, (r, t, c, float(err))
        torch.testing.assert_close(got, want, atol=2e-2, rtol=2e-2)
        off += t
    from vllm_b200 import capi
    assert capi.device_status() == 0


@pytest.mark.parametrize("D", [32, 64, 80, 96, 112, 120, 128, 192, 256])
@pytest.mark.parametrize("kv,dtype", [("auto", torch.bfloat16), ("auto", torch.float16),
                                      ("fp8", torch.bfloat16), ("fp8_e5m2", torch.float16)])
@pytest.mark.parametrize("B", [16, 32])
def test_head_sizes_types_and_blocks(D, kv, dtype, B):
    if D == 120 and kv != "auto":
        pytest.skip("an fp8 cache keeps 16 head dimensions together")
    _case([1, 1, 70, 3, 200], [5, 300, 0, 129, 61], 8, 2, D, B, dtype, kv, alibi=D == 96, seed=D)


# row tiles hold 128 // (H // HK) tokens, two to an item; key tiles 128 (64 above head size 128)
@pytest.mark.parametrize("H,HK", [(4, 4), (12, 4), (28, 4), (32, 2), (33, 1)])
@pytest.mark.parametrize("q,ctx", [(2, 0), (15, 1), (16, 112), (17, 112), (31, 97), (127, 1), (128, 0),
                                   (129, 127), (255, 2), (256, 128), (257, 511)])
def test_tile_edges(H, HK, q, ctx):
    _case([q, 0, q], [ctx, 7, 0], H, HK, 128, 16, torch.bfloat16, "auto", seed=q)


@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_strides_of_dimensions_of_size_one(kv):
    """One token, one kv head, one block: whatever strides these come with, the prefill kernel takes the call."""
    from vllm_b200 import _custom_ops as ops
    H, D, B, n, x = 4, 128, 16, 11, 8 if kv == "auto" else 16
    gen = torch.Generator(device=DEV).manual_seed(0)
    kc, vc = torch.randn(D // x, B, x, generator=gen, device=DEV), torch.randn(D, B, generator=gen, device=DEV)
    kc, vc = (t.bfloat16() if kv == "auto" else t.to(torch.float8_e4m3fn).view(torch.uint8) for t in (kc, vc))
    q = torch.randn(H, D, generator=gen, device=DEV).bfloat16()
    out = torch.full((1, H, D), float("nan"), dtype=q.dtype, device=DEV)
    table, lens, qsl = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([[0]], [n], [0, 1]))
    one = torch.tensor(1.0, device=DEV)
    assert ops.paged_attention_varlen(out, q.as_strided((1, H, D), (0, D, 1)),
                                      kc.as_strided((1, 1, D // x, B, x), (0, 0, B * x, x, 1)),
                                      vc.as_strided((1, 1, D, B), (0, 0, B, 1)), 1, D ** -0.5, table, lens, qsl, 0, B, n,
                                      None, kv, one, one)
    k, v = _gather(kc[None, None], vc[None, None], table[0], n, kv, 1.0)
    want = torch.softmax(q.float() @ k[:, 0].T * D ** -0.5, -1) @ v[:, 0]
    assert (out[0].float() - want).norm() < 6e-3 * want.norm()  # (P and the result are rounded to 16 bits)


# V comes in pages of 16 keys: the last one of a sequence is cut at every length, the pages behind it do not exist
@pytest.mark.parametrize("D", [64, 120, 192])
@pytest.mark.parametrize("B", [16, 32])
def test_sequences_that_end_anywhere_in_a_page(D, B):
    _case([3 + i % 7 for i in range(40)], [110 + i for i in range(40)], 8, 2, D, B, torch.bfloat16, "auto", seed=B)


@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_few_rows_behind_long_contexts_are_split(kv):
    _case([5, 2, 40], [9000, 3000, 20000], 8, 2, 128, 16, torch.bfloat16, kv)


def test_merges_of_cut_rows_launch_after_launch():
    """The pieces of a row meet in the same workspace in every launch: with other queries each time, and no
    host in between, a merge that read a piece of the launch before it would give that launch's values."""
    from vllm_b200 import _custom_ops as ops
    H, HK, D, B, T, n, runs = 8, 2, 128, 16, 64, 8256, 24
    gen = torch.Generator(device=DEV).manual_seed(1)
    kc = torch.randn(n // B, HK, D // 8, B, 8, generator=gen, device=DEV).bfloat16()
    vc = torch.randn(n // B, HK, D, B, generator=gen, device=DEV).bfloat16()
    q = (4 * torch.randn(runs, T, H, D, generator=gen, device=DEV)).bfloat16()
    out = torch.full_like(q, float("nan"))
    table = torch.randperm(n // B, generator=gen, device=DEV).int().view(1, -1)
    lens, qsl = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in ([n], [0, T]))
    one = torch.tensor(1.0, device=DEV)
    for i in range(runs):
        assert ops.paged_attention_varlen(out[i], q[i], kc, vc, HK, D ** -0.5, table, lens, qsl, 0, B, n, None,
                                          "auto", one, one)
    k, v = _gather(kc, vc, table[0], n, "auto", 1.0)
    hidden = torch.arange(n, device=DEV).view(1, -1) > torch.arange(n - T, n, device=DEV).view(-1, 1)
    for i in range(runs):
        s = torch.einsum("tkgd,lkd->kgtl", q[i].float().view(T, HK, H // HK, D), k) * D ** -0.5
        want = torch.einsum("kgtl,lkd->tkgd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), v)
        # (P, the partials and the result are rounded to 16 bits: 2^-9 each)
        assert (out[i].float() - want.reshape(T, H, D)).norm() < 6e-3 * want.norm(), i


def test_many_requests_and_single_rows_among_them():
    rng = np.random.default_rng(3)
    q = rng.integers(1, 40, size=600)  # (512 requests to a launch)
    q[:20] = 1
    q[100] = 1
    _case(q, rng.integers(0, 400, size=600), 8, 2, 64, 16, torch.bfloat16, "auto")


@pytest.mark.parametrize("kv,dtype", [("auto", torch.bfloat16), ("fp8_e5m2", torch.bfloat16), ("fp8", torch.float16)])
@pytest.mark.parametrize("alibi", [False, True])
@pytest.mark.parametrize("HK", [2, 8])
def test_short_chunks_with_and_without_bias(kv, dtype, alibi, HK):
    _case([37, 120, 203, 25, 108, 191, 96, 179, 300], [16, 17, 18, 13, 14, 15, 11, 12, 400], 32, HK, 128, 16,
          dtype, kv, alibi=alibi)


@pytest.mark.parametrize("kv", ["auto", "fp8"])
@pytest.mark.parametrize("alibi", [False, True])
def test_items_whose_second_row_tile_is_empty(kv, alibi):
    # (the warpgroup of the second row tile runs items ahead of everybody else)
    _case([20 + i % 12 + 64 * (i % 3) for i in range(60)], [i % 19 for i in range(60)], 32, 8, 128, 16,
          torch.bfloat16, kv, alibi=alibi)


# A row's running maximum is only raised when a tile shows that it is too low: in its first half (sum of the
# exponentials) or its second (their maximum)
@pytest.mark.parametrize("kv,dtype", [("auto", torch.bfloat16), ("auto", torch.float16), ("fp8", torch.bfloat16)])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("ramp", [0.02, 0.3])
def test_maxima_that_grow_along_the_sequence(kv, dtype, D, ramp):
    _case([130, 40, 300], [0, 700, 333], 8, 2, D, 16, dtype, kv, ramp=ramp)


# Keys with a logit of -inf leave a row without a maximum; whole key tiles of them, and 1 to 20 finite low logits
# in the first half of the tiles behind
@pytest.mark.parametrize("kv,dtype", [("auto", torch.bfloat16), ("auto", torch.float16), ("fp8_e5m2", torch.bfloat16)])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("alibi", [False, True])
@pytest.mark.parametrize("q,ctx", [([1, 20], [128, 148]), ([40, 2, 3], [300, 257, 128]), ([5, 30], [9000, 3100])],
                         ids=["few-finite", "whole", "cut"])
@pytest.mark.parametrize("first,low", [(128, -60.0), (256, -8.0)])
def test_keys_of_minus_infinity(kv, dtype, D, alibi, q, ctx, first, low):
    _case(q, ctx, 8, 2, D, 16, dtype, kv, alibi=alibi, dark=(first, low))


@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_a_long_prompt(kv):
    _case([1500, 900], [700, 0], 8, 2, 128, 16, torch.bfloat16, kv)


# The workspace has 496 slots for pieces on the first stream of a process, 62 on any other, half of them
# beside a decode launch: what is cut has to fit, and what is not cut must not count.
@pytest.mark.parametrize("decodes", [0, 5])
@pytest.mark.parametrize("stream", ["first", "second"])
@pytest.mark.parametrize("kv", ["auto", "fp8"])
def test_long_contexts_are_cut_beside_many_whole_groups(kv, stream, decodes):
    rng = np.random.default_rng(decodes)
    q = np.concatenate([[1] * decodes, [16], rng.integers(2, 65, size=40), [9, 70], rng.integers(2, 65, size=20)])
    ctx = rng.integers(0, 700, size=len(q))
    ctx[decodes], ctx[decodes + 41], ctx[decodes + 42] = 20000, 5000, 900
    with torch.cuda.stream(torch.cuda.current_stream() if stream == "first" else torch.cuda.Stream()):
        _case(q.astype(int), ctx, 32, 8, 128, 16, torch.bfloat16, kv, seed=decodes)


def test_a_long_context_does_not_run_on_one_sm_beside_many_groups():
    """Cut into pieces it takes about as long beside 480 other groups as they and it take apart; as one
    item per kv head it took three times as long."""
    from vllm_b200 import _custom_ops as ops
    H, HK, D, B, pool = 32, 8, 128, 16, 2048
    kc = torch.randn(pool, HK, D // 8, B, 8, device=DEV).bfloat16()
    vc = torch.randn(pool, HK, D, B, device=DEV).bfloat16()
    one = torch.tensor(1.0, device=DEV)

    def time(q, lens):
        n = sum(q)
        query = torch.randn(n, H, D, device=DEV).bfloat16()
        out = torch.empty_like(query)
        table = torch.randint(0, pool, (len(q), -(-max(lens) // B)), dtype=torch.int32, device=DEV)
        qsl = torch.tensor(np.concatenate([[0], np.cumsum(q)]), dtype=torch.int32, device=DEV)
        seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                assert ops.paged_attention_varlen(out, query, kc, vc, HK, D ** -0.5, table, seq_lens, qsl, 0, B,
                                                  max(lens), None, "auto", one, one)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    long, others = ([16], [32016]), ([32] * 60, [1000] * 60)
    both = time(long[0] + others[0], long[1] + others[1])
    assert both < 1.5 * (time(*long) + time(*others))
