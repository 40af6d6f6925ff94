"""The direct bindings of _custom_ops: whatever has to see an operator - tracers, dispatch modes, the
profiler, function transforms, the operators' own checks - sees it as through torch.ops."""
import pytest
import torch

from vllm_b200 import _custom_ops as ops
import workloads as W

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _write_args():
    gen = torch.Generator(device=DEV).manual_seed(0)
    k, v = (torch.randn(5, 2, 64, generator=gen, device=DEV).bfloat16() for _ in range(2))
    kc = torch.zeros(4, 2, 8, 16, 8, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros(4, 2, 64, 16, dtype=torch.bfloat16, device=DEV)
    slots = torch.tensor([3, 17, 40, 41, 63], device=DEV)
    one = torch.tensor(1.0, device=DEV)
    return k, v, kc, vc, slots, one


def _write(k, v, kc, vc, slots, one):
    ops.reshape_and_cache(k, v, kc, vc, slots, "auto", one, one)
    return kc


def test_a_dispatch_mode_sees_the_operators():
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    args = _write_args()
    with Record():
        _write(*args)
    assert seen == ["_C_b200_cache_ops.reshape_and_cache.default"]
    assert args[2].any()


def test_the_profiler_sees_the_operators():
    from torch.profiler import ProfilerActivity, profile
    w = W.small(DEV, num_seqs=2, max_len=100, num_blocks=64)
    with profile(activities=[ProfilerActivity.CPU]) as prof:
        W.run_attention(w, version="v1")
        _write(*_write_args())
    names = {e.key for e in prof.key_averages()}
    assert {"_C_b200::paged_attention_v1", "_C_b200_cache_ops::reshape_and_cache"} <= names


def test_tracing_does_not_lose_an_operator():
    """torch.jit.trace refuses these schemas (anonymous alias sets); it must not record a graph without
    the write instead."""
    k, v, kc, vc, slots, one = _write_args()

    def through(write):
        def f(k, v, kc, vc):
            write(k, v, kc, vc, slots, "auto", one, one)
            return kc
        return f
    for write in (torch.ops._C_b200_cache_ops.reshape_and_cache, ops.reshape_and_cache):
        try:
            traced = torch.jit.trace(through(write), (k, v, kc, vc), check_trace=False)
        except RuntimeError:
            continue
        assert "reshape_and_cache" in str(traced.graph)


def test_a_compiled_function_keeps_its_operators():
    eager, compiled = _write_args(), _write_args()
    _write(*eager)
    torch.compile(_write, fullgraph=True, backend="eager")(*compiled)
    assert torch.equal(eager[2], compiled[2]) and torch.equal(eager[3], compiled[3]) and eager[2].any()


def test_function_transforms_are_refused_as_by_the_operators():
    k, v, kc, vc, slots, one = _write_args()
    batch = [t.unsqueeze(0).repeat(2, *[1] * t.dim()) for t in (k, v, kc, vc)]

    def through(write):
        def f(k, v, kc, vc):
            write(k, v, kc, vc, slots, "auto", one, one)
            return kc
        return f
    for write in (torch.ops._C_b200_cache_ops.reshape_and_cache, ops.reshape_and_cache):
        with pytest.raises(RuntimeError):
            torch.vmap(through(write))(*batch)
    assert not batch[2].any()


@pytest.mark.parametrize("spoil", ["slots dtype", "cpu cache", "kv type", "cache dtype", "strided heads"])
def test_wrong_arguments_raise_what_the_operators_raise(spoil):
    k, v, kc, vc, slots, one = _write_args()
    kv = "auto"
    if spoil == "slots dtype":
        slots = slots.int()
    elif spoil == "cpu cache":
        kc = kc.cpu()
    elif spoil == "kv type":
        kv = "int3"
    elif spoil == "cache dtype":
        kc = kc.half()
    else:
        k = torch.zeros(5, 4, 64, dtype=torch.bfloat16, device=DEV)[:, ::2]
    errors = []
    for write in (torch.ops._C_b200_cache_ops.reshape_and_cache, ops.reshape_and_cache):
        with pytest.raises((RuntimeError, NotImplementedError)) as e:
            write(k, v, kc, vc, slots, kv, one, one)
        errors.append((type(e.value), str(e.value).splitlines()[0]))
    assert errors[0] == errors[1]
    assert not vc.any()
