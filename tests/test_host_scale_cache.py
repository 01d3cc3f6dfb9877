"""The cache of swizzled weight scales in the native host path (csrc/host.cpp), which all threads share."""

import gc
import threading
import time

import pytest
import torch

from flashim_b200 import _native
from flashim_b200.backends.sm100 import kernels
from flashim_b200.quant import swizzle_scales

ENTRIES = 512


@pytest.fixture()
def bound():
    """``bind(swizzle)``: the module with that function in place of ``swizzle_scales``."""
    if not _native.available():
        pytest.skip("the native libraries are not built")
    module = kernels._host()

    def bind(swizzle):
        module.bind(str(_native.LIBRARY_PATH), lambda index: None, _native.check, None, swizzle, kernels.QuantizedTensor, kernels.Int8Tensor)
        return module

    yield bind
    kernels._host.cache_clear()
    kernels._host()


def exponents(fill, rows=32):
    return torch.full((rows, 4), fill, dtype=torch.int8)


def test_two_misses_on_one_key_leave_one_entry(bound):
    """The swizzle may let another thread in, which misses on the same tensor: the entry that stays must survive 511 others."""
    e, calls = exponents(3), []

    def swizzle(t):
        calls.append(t.data_ptr())
        if calls.count(e.data_ptr()) == 1:
            module.swizzled_scales(e)  # what the other thread does meanwhile
        return swizzle_scales(t)

    module = bound(swizzle)
    want = swizzle_scales(e)
    assert torch.equal(module.swizzled_scales(e), want) and calls.count(e.data_ptr()) == 2
    others = [exponents(i % 100) for i in range(ENTRIES - 1)]
    for other in others:
        module.swizzled_scales(other)
    assert torch.equal(module.swizzled_scales(e), want) and calls.count(e.data_ptr()) == 2


def test_entry_follows_its_tensor(bound):
    calls = []
    module = bound(lambda t: (calls.append(1), swizzle_scales(t))[1])
    e = exponents(1)
    first = module.swizzled_scales(e)
    assert module.swizzled_scales(e) is not None and len(calls) == 1
    e.fill_(2)
    assert torch.equal(module.swizzled_scales(e), swizzle_scales(e)) and len(calls) == 2
    assert torch.equal(first, swizzle_scales(exponents(1)))  # what a caller holds stays as it was
    others = [exponents(i % 100) for i in range(ENTRIES)]
    for other in others:
        module.swizzled_scales(other)
    module.swizzled_scales(e)
    assert len(calls) == 2 + ENTRIES + 1  # the least recently used one went


@pytest.mark.gpu
def test_two_threads_and_an_exponent_that_changes_in_place():
    """One thread rewrites the exponents in place (the same values, a new version) and calls, the other only calls: each call has to
    keep the scales that it looked up while the other takes their entry out."""
    import flashim_b200
    from flashim_b200.quant import QuantizedTensor, QuantizedWeight

    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    up, down = QuantizedWeight.from_float(rand(256, 128) * 0.1), QuantizedWeight.from_float(rand(128, 256) * 0.1)
    x = QuantizedTensor((rand(96, 128) * 16).to(torch.float8_e4m3fn), torch.full((4,), -6, dtype=torch.int8, device="cuda"), (96, 128))
    hidden, bias, out = torch.full((8,), -4, dtype=torch.int8, device="cuda"), rand(256).bfloat16(), rand(256).bfloat16()
    conv = (x.values.view(1, 8, 12, 128), x.scale_exponent, up.values, up.scale_exponent, out, 1, 1, 1, 1, 0, 0, 1, 1)
    ops = flashim_b200.ops

    def call():
        return [ops.mxfp8_linear(x, out, up), ops.mxfp8_gelu_mlp(x, up, bias, hidden, down), ops.mxfp8_conv2d(*conv)]

    want, wrong = call(), []

    def work(change):
        for _ in range(300):
            if change:
                up.scale_exponent.add_(0), down.scale_exponent.add_(0)
            got = call()
            if not all(torch.equal(a, b) for a, b in zip(got, want)):
                wrong.append(change)

    threads = [threading.Thread(target=work, args=(change,)) for change in (True, False)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not wrong
    ops.reset_call_counts()


def linear(seed, rows=96):
    from flashim_b200.quant import QuantizedTensor, QuantizedWeight

    g = torch.Generator(device="cuda").manual_seed(seed)
    weight = QuantizedWeight.from_float(torch.randn(256, 128, generator=g, device="cuda") * 0.1)
    x = torch.randn(rows, 128, generator=g, device="cuda").to(torch.float8_e4m3fn)
    return QuantizedTensor(x, torch.zeros(4, dtype=torch.int8, device="cuda"), (rows, 128)), torch.zeros(256, dtype=torch.bfloat16, device="cuda"), weight


def expected(x, bias, weight):
    return (x.dequantize().double() @ weight.dequantize().double().t()).float()


def evict():
    for _ in range(ENTRIES):
        kernels._host().swizzled_scales(exponents(1))


@pytest.mark.gpu
def test_graph_keeps_the_scales_that_it_reads():
    """The entry goes while the graph lives: the graph reads the same scales, and their memory comes back once it has gone."""
    from flashim_b200 import ops

    args = linear(2)
    want = ops.mxfp8_linear(*args)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.mxfp8_linear(*args)
    evict()
    others = [torch.full((1024,), 255, dtype=torch.uint8, device="cuda") for _ in range(64)]  # (256 x 128 weights have 1 KB of scales)
    out.zero_()
    graph.replay()
    assert torch.equal(out, want) and len(others) == 64
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    del graph
    gc.collect()
    deadline = time.monotonic() + 10
    while torch.cuda.memory_allocated() >= held and time.monotonic() < deadline:
        evict()
    assert torch.cuda.memory_allocated() < held
    ops.reset_call_counts()


@pytest.mark.gpu
def test_first_use_inside_a_capture():
    """Scales that only the graph's replays form are not there for calls outside of it."""
    from flashim_b200 import ops

    ops.mxfp8_linear(*linear(3))  # (kernels loaded)
    args = linear(4)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.mxfp8_linear(*args)
    got = ops.mxfp8_linear(*args)
    assert float((got.float() - expected(*args)).norm() / expected(*args).norm()) < 4e-3  # (one bf16 rounding: 2**-9 at most)
    graph.replay()
    assert torch.equal(out, got)
    ops.reset_call_counts()


BUSY = 200_000_000  # clock ticks: a tenth of a second and more


@pytest.fixture()
def streams():
    """Two streams with memory of their own, and calls that do not read the status word (which would wait for them)."""
    from flashim_b200 import ops

    kernels._host().bind(str(_native.LIBRARY_PATH), lambda index: kernels.status_word(torch.device("cuda", index)), _native.check, None,
                         swizzle_scales, kernels.QuantizedTensor, kernels.Int8Tensor)
    pair = torch.cuda.Stream(), torch.cuda.Stream()
    for stream in pair:
        with torch.cuda.stream(stream):
            ops.mxfp8_linear(*linear(6))
    torch.cuda.synchronize()
    yield pair
    torch.cuda.synchronize()
    kernels._host.cache_clear()
    kernels._host()
    ops.reset_call_counts()


@pytest.mark.gpu
def test_a_stream_waits_for_the_scales_of_another(streams):
    """The kernels that form the scales stand behind a long one on their stream; a call on a second stream finds the entry meanwhile."""
    from flashim_b200 import ops

    args, (first, second) = linear(5), streams
    want = expected(*args)
    torch.cuda.synchronize()
    with torch.cuda.stream(first):
        torch.cuda._sleep(BUSY)
        here = ops.mxfp8_linear(*args)
    with torch.cuda.stream(second):
        there = ops.mxfp8_linear(*args)
    assert not first.query()
    torch.cuda.synchronize()
    assert torch.equal(here, there) and float((here.float() - want).norm() / want.norm()) < 4e-3  # (one bf16 rounding)


@pytest.mark.gpu
def test_memory_of_scales_that_another_stream_reads(streams):
    """The entry goes while a call on a second stream has yet to read its scales: the first stream must not get their memory."""
    from flashim_b200 import ops

    args, (first, second) = linear(7), streams
    with torch.cuda.stream(first):
        want = ops.mxfp8_linear(*args)
    torch.cuda.synchronize()
    with torch.cuda.stream(second):
        torch.cuda._sleep(BUSY)
        got = ops.mxfp8_linear(*args)
    evict()
    with torch.cuda.stream(first):
        others = [torch.full((1024,), 255, dtype=torch.uint8, device="cuda") for _ in range(64)]
    assert not second.query() and len(others) == 64
    torch.cuda.synchronize()
    assert torch.equal(got, want)
