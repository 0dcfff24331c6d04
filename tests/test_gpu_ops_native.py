"""The two ops through their native registration against the same calls through the Python one, which inference mode takes."""

import ctypes
import threading

import pytest
import torch

from megabake_b200 import CompilerError, _native, ops  # noqa: F401
from megabake_b200.runtime import AttentionKernels
from megabake_b200.synth import synth_normal

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


def _tensor(name, *shape):
    return synth_normal(shape, seed=31, name=name, std=1.0, device=DEVICE)


def _kv_case(batch, heads, kv_heads, dim, filled, capacity, strided):
    def vector(name, n):
        if strided:  # as a model hands them over: [batch, heads, 1, dim], transposed
            return _tensor(name, batch, n, 1, dim).transpose(1, 2)
        return _tensor(name, batch, 1, n, dim)
    caches = [_tensor(name, batch, capacity, kv_heads, dim) for name in ("kc", "vc")]
    return [vector("q", heads), vector("k", kv_heads), vector("v", kv_heads), *caches,
            torch.full((1,), filled, dtype=torch.int32, device=DEVICE)]


@pytest.mark.parametrize("shape", [(1, 4, 4, 64, 0, 1), (3, 8, 2, 128, 17, 40), (20, 9, 3, 64, 300, 301)])
@pytest.mark.parametrize("strided", [False, True])
def test_decode_op_is_the_same_on_both_routes(shape, strided):
    for _ in range(2):  # the first call makes the handle, on the Python route in any case
        mine, theirs = _kv_case(*shape, strided), _kv_case(*shape, strided)
        versions = [t._version for t in mine]
        out = torch.ops.megabake.kv_attention(*mine)
        with torch.inference_mode():
            expected = torch.ops.megabake.kv_attention(*theirs)
        assert torch.equal(out, expected) and all(torch.equal(a, b) for a, b in zip(mine, theirs))
        assert [t._version - v for t, v in zip(mine, versions)] == [0, 0, 0, 1, 1, 1]


@pytest.mark.parametrize("shape", [(1, 4, 4, 64, 1, 1), (2, 8, 2, 128, 65, 130), (40, 9, 3, 64, 33, 33)])
@pytest.mark.parametrize("mask", [None, "plain", "expanded", "float"])
def test_prompt_op_is_the_same_on_both_routes(shape, mask):
    batch, heads, kv_heads, dim, queries, keys = shape
    q, k, v = _tensor("q", batch, queries, heads, dim), _tensor("k", batch, keys, kv_heads, dim), _tensor("v", batch, keys, kv_heads, dim)
    m = None if mask is None else _tensor("m", 1 if mask == "expanded" else batch, 1, queries, keys)
    m = m.expand(batch, 1, queries, keys) if mask == "expanded" else (m.float() if mask == "float" else m)
    for _ in range(2):
        out = torch.ops.megabake.attention(q, k, v, m, dim ** -0.5)
        with torch.inference_mode():
            expected = torch.ops.megabake.attention(q, k, v, m, dim ** -0.5)
        assert torch.equal(out, expected)


@pytest.mark.parametrize("keys", [48, 333, 512])
def test_a_mask_written_by_the_kernel_right_before(keys):
    """The op's kernel begins while that one is at work: every call sees its own mask."""
    q, k, v = (_tensor(name, 1, keys, 8, 64) for name in ("a", "b", "c"))
    masks = [_tensor(f"m{i}", 1, 1, keys, keys) for i in range(4)]
    expected = [torch.ops.megabake.attention(q, k, v, m, 0.125) for m in masks]
    mask = torch.empty_like(masks[0])
    torch.cuda.synchronize()
    results = []
    for _ in range(10):
        for m in masks:
            mask.copy_(m)
            results.append(torch.ops.megabake.attention(q, k, v, mask, 0.125))
    assert all(torch.equal(r, expected[i % 4]) for i, r in enumerate(results))


def test_what_the_ops_refuse_is_refused_on_both_routes():
    good = _kv_case(2, 4, 2, 64, 3, 8, False)
    torch.ops.megabake.kv_attention(*good)
    for index, wrong in ((0, good[0].half()), (0, good[0].expand(2, 1, 4, 64).repeat(1, 2, 1, 1)), (3, good[3].transpose(0, 1)),
                         (5, good[5].long())):
        args = list(good)
        args[index] = wrong
        errors = []
        for mode in (torch.no_grad(), torch.inference_mode()):
            with mode, pytest.raises(Exception) as caught:
                torch.ops.megabake.kv_attention(*args)
            errors.append((type(caught.value), str(caught.value)))
        assert errors[0] == errors[1]
    full = _kv_case(2, 4, 2, 64, 8, 8, False)
    assert torch.isnan(torch.ops.megabake.kv_attention(*full)).all()
    torch.cuda.synchronize()
    with pytest.raises(CompilerError, match="state-capacity|exceeds capacity"):
        torch.ops.megabake.kv_attention(*_kv_case(2, 4, 2, 64, 3, 8, False))


def test_a_result_that_wants_a_gradient_says_that_there_is_none():
    args = _kv_case(2, 4, 2, 64, 3, 8, False)
    args[0].requires_grad_(True)
    prompt = [_tensor(name, 1, 8, 4, 64).requires_grad_(True) for name in ("a", "b", "c")]
    for out in (torch.ops.megabake.kv_attention(*args), torch.ops.megabake.attention(*prompt, None, 0.125)):
        assert out.requires_grad
        with pytest.raises(RuntimeError, match="no autograd formula was registered"):
            out.float().sum().backward()


def test_standard_calls_do_not_reach_python(monkeypatch):
    """Once a head shape has its handle: without this the equality of the two routes above could be that of one route."""
    cases = [_kv_case(3, 8, 2, 128, 17, 40, strided) for strided in (False, True)]
    prompt = [_tensor("q", 2, 65, 8, 128), _tensor("k", 2, 130, 2, 128), _tensor("v", 2, 130, 2, 128)]
    mask = _tensor("m", 2, 1, 65, 130)
    torch.ops.megabake.kv_attention(*_kv_case(3, 8, 2, 128, 17, 40, False))

    def never(*args):
        raise AssertionError("the Python route")

    monkeypatch.setattr(AttentionKernels, "kv_attention", never)
    monkeypatch.setattr(AttentionKernels, "attention", never)
    for args in cases:
        torch.ops.megabake.kv_attention(*args)
    for m in (None, mask):
        torch.ops.megabake.attention(*prompt, m, 0.1)
    with torch.inference_mode(), pytest.raises(AssertionError, match="the Python route"):
        torch.ops.megabake.attention(*prompt, None, 0.1)


def test_a_call_does_not_wait_for_one_of_another_head_shape():
    """The library's entry for one shape is replaced by one that waits; meanwhile a call of another shape comes and goes."""
    slow, quick = ([_tensor(name, 1, 80, heads, 64) for name in ("a", "b", "c")] for heads in (15, 12))
    expected = [torch.ops.megabake.attention(*args, None, 0.125) for args in (slow, quick)][1]
    kernels = AttentionKernels.for_shape(15, 15, 64, 1, DEVICE)
    entered, go_on = threading.Event(), threading.Event()

    @ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_void_p] * 5, ctypes.c_float, *[ctypes.c_int] * 3, ctypes.c_void_p, ctypes.c_void_p)
    def waits(*args):
        entered.set()
        go_on.wait(20)
        return _native.MK_OK  # (its result is memory as it was allocated, and not looked at)

    def register(entry):
        lib = _native.load()
        entries = [ctypes.cast(e, ctypes.c_void_p) for e in (lib.mk_kv_attention_scratch, lib.mk_kv_attention_scratch_bytes, entry)]
        _native._ops_library.megabake_ops_register(15, 15, 64, 0, kernels.max_tokens, kernels._handle, kernels._mirror.data_ptr(), *entries)

    register(waits)
    thread = threading.Thread(target=lambda: torch.ops.megabake.attention(*slow, None, 0.125))
    try:
        thread.start()
        assert entered.wait(20)
        out = torch.ops.megabake.attention(*quick, None, 0.125)
        assert thread.is_alive() and torch.equal(out, expected)
    finally:
        go_on.set()
        thread.join()
        register(_native.load().mk_attention)


def test_a_captured_prompt_op_outlives_longer_prompts_and_larger_batches():
    """What a graph's launches point to stays where it is: memory that was free for others is written over before the replay."""
    shape = (5, 5, 64)
    args = [_tensor(name, 1, 200, 5, 64) for name in ("a", "b", "c")]
    expected = torch.ops.megabake.attention(*args, None, 0.125)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = torch.ops.megabake.attention(*args, None, 0.125)
    first = AttentionKernels.for_shape(*shape, 1, DEVICE)
    torch.ops.megabake.attention(*[_tensor(name, 4, 900, 5, 64) for name in ("a", "b", "c")], None, 0.125)
    assert AttentionKernels.for_shape(*shape, 1, DEVICE) is first  # a prompt of any length has room
    torch.ops.megabake.kv_attention(*_kv_case(70, *shape, 17, 40, False))
    assert AttentionKernels.for_shape(*shape, 1, DEVICE) is not first and first in AttentionKernels._superseded
    torch.cuda.synchronize()
    blocks = [torch.full((1 << 20,), -1, dtype=torch.int32, device=DEVICE) for _ in range(64)]
    out.zero_()
    graph.replay()
    assert torch.equal(out, expected) and (first.workspace[:16] != 255).any()
    del blocks


def test_decode_op_in_a_captured_graph_and_on_two_streams():
    expected = torch.ops.megabake.kv_attention(*_kv_case(3, 8, 2, 128, 17, 40, False))
    args, start = _kv_case(3, 8, 2, 128, 17, 40, False), torch.full((1,), 17, dtype=torch.int32, device=DEVICE)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert torch.equal(torch.ops.megabake.kv_attention(*args), expected)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        args[5].copy_(start)
        out = torch.ops.megabake.kv_attention(*args)
    for _ in range(2):
        out.zero_()
        graph.replay()
        assert torch.equal(out, expected)
