"""The native call of each op (csrc/host.cpp): the bytes of the Python implementation for the calls it takes, and
``NotImplemented`` for those that the general path has to convert, record or refuse."""

import pytest
import torch

from fim_testlib import DEV, same_bytes

pytestmark = pytest.mark.gpu
BF16, E4M3 = torch.bfloat16, torch.float8_e4m3fn
K3 = (3, 3, 1, 1, 1, 1, 1, 1)


@pytest.fixture(scope="module")
def ops():
    import flashim_b200

    yield flashim_b200.ops
    flashim_b200.ops.reset_call_counts()  # other modules count calls


def _calls(ops):
    """One call per op: name -> (args, kwargs)."""
    from flashim_b200.quant import QuantizedTensor, QuantizedWeight, swizzle_scales
    from flashim_b200.quant.tensor import int8_weight_from_conv

    g = torch.Generator(device=DEV).manual_seed(5)
    rand = lambda *s, dtype=torch.float32: torch.randn(s, generator=g, device=DEV).to(dtype)  # noqa: E731
    x = rand(2, 9, 11, 128, dtype=BF16)
    e, oe = torch.full((4,), -6, dtype=torch.int8, device=DEV), torch.full((4,), -4, dtype=torch.int8, device=DEV)
    bias, scale = rand(128, dtype=BF16), torch.tensor(0.03, device=DEV)
    w3, w1 = QuantizedWeight.from_conv(rand(128, 128, 3, 3) * 0.05), QuantizedWeight.from_conv(rand(128, 128, 1, 1) * 0.1)
    i3, i3s = int8_weight_from_conv(rand(128, 128, 3, 3))
    i1, i1s = int8_weight_from_conv(rand(128, 128, 1, 1))
    up, down = QuantizedWeight.from_float(rand(256, 128) * 0.1), QuantizedWeight.from_float(rand(128, 256) * 0.1)
    res, image = rand(2, 9, 11, 128, dtype=BF16), x.permute(0, 3, 1, 2)
    q, xi = (x.float() * 16).to(E4M3), torch.randint(-127, 128, x.shape, generator=g, device=DEV, dtype=torch.int8)
    qd, qs = ops.quantize_mxfp8_dynamic(x)
    qt = QuantizedTensor(q.view(-1, 128), e, (198, 128))
    dw, db = rand(25, 128, dtype=BF16), rand(128)
    mlp = (qd, qs, up.values, up.swizzled_scales(), rand(256, dtype=BF16), down.values, down.swizzled_scales(), bias, res)
    f, warp = rand(2, 5, 7, 32), rand(2, 5, 7, 2)
    return {
        "quantize_mxfp8": ((x, e), {}), "quantize_int8": ((x, scale), {}), "quantize_mxfp8_dynamic": ((x,), {}),
        "gelu_quantize": ((x, e), {"input_bias": db}),
        "mxfp8_conv2d": ((q, e, w3.values, w3.scale_exponent, bias, *K3), {"relu": True, "residual": res, "out_exponent": oe}),
        "mxfp8_conv2d_fused": ((q, e, w3.values, w3.swizzled_scales(), bias, *K3), {"act": "gelu", "dynamic_out": True}),
        "mxfp8_conv2d_bf16": ((x, None, w1.values, swizzle_scales(w1.scale_exponent), bias), {"out_fp32": True}),
        "mxfp8_gelu_mlp_residual": (mlp, {}),
        "int8_conv2d": ((xi, i3, scale, i3s, bias, *K3), {"residual": res, "out_scale": scale}),
        "int8_conv2d_maxpool": ((xi, i3, scale, i3s, None, *K3), {"relu": True, "out_scale": scale}),
        "mxfp8_linear": ((qt, bias, w1), {}), "mxfp8_gelu_mlp": ((qt, up, rand(256, dtype=BF16), oe.repeat(2), down), {}),
        "mxfp8_scaled_mm": ((qd.view(-1, 128), w1.values.t(), qs, w1.swizzled_scales()), {"bias": bias}),
        "int8_linear": ((xi.view(-1, 128), i1, scale, i1s, bias), {"gelu": True, "residual": res.view(-1, 128)}),
        "depthwise5x5_act": ((image, dw, db), {"act": "relu"}), "depthwise5x5_act_mxfp8": ((image, dw, db), {}),
        "depthwise5x5_relu_mxfp8": ((image, dw, db), {}), "depthwise5x5_relu_int8": ((image, dw, db, scale), {}),
        "depthwise5x5_relu_pointwise": ((image, dw, db, rand(64, 128, dtype=BF16), bias[:64]), {}),
        "depthwise5x5_relu_pointwise_mxfp8": ((image, dw, db, w1.values, w1.swizzled_scales(), None, bias), {}),
        "depthwise5x5_relu_pointwise_int8": ((image, dw, db, i1, i1s, bias, scale), {}),
        "romav2_refiner_input": ((f, f, warp, rand(8, 2), rand(8), (3.0, 2.0), 2), {"pair": 1}),
        "romav2_refiner_heads": ((image, rand(6, 128), rand(6), rand(2, 9, 11, 2), rand(2, 9, 11, 1), 4.0), {}),
    }


def _leaves(out):
    if isinstance(out, torch.Tensor):
        return [out]
    if isinstance(out, tuple):
        return [t for part in out for t in _leaves(part)]
    return _leaves(tuple(v for v in vars(out).values() if isinstance(v, torch.Tensor)))


def test_native_calls_give_the_bytes_of_the_python_implementations(ops):
    for name, (args, kwargs) in _calls(ops).items():
        op = getattr(ops, name)
        assert op._direct is not None and op._direct[0] == "sm100", name
        got, want = op._direct[1](*args, **kwargs), op.impls[0].fn(*args, **kwargs)
        assert got is not NotImplemented and type(got) is type(want), name
        for a, b in zip(_leaves(got), _leaves(want), strict=True):
            assert a.dtype == b.dtype and a.stride() == b.stride() and same_bytes(a, b), name
        if hasattr(want, "logical_shape"):
            assert got.logical_shape == want.logical_shape
        assert op(*args, **kwargs) is not NotImplemented


def test_calls_for_the_general_path(ops):
    calls = _calls(ops)
    x, e = calls["quantize_mxfp8"][0]
    direct = ops.quantize_mxfp8._direct[1]
    assert direct(x[:, :, 1:], e) is NotImplemented                      # strided
    assert direct(x.half(), e) is NotImplemented                         # a dtype the op has no kernel for
    assert direct(x.flatten()[1:129].view(1, 128), e) is NotImplemented  # not 16-byte aligned: the wrapper copies
    assert direct(x.clone().requires_grad_(), e) is NotImplemented       # autograd records
    assert direct(x, e, 1) is NotImplemented and direct(x, exponent=e) is NotImplemented
    assert torch.func.vmap(lambda v: direct(v, e) is NotImplemented and v)(x) is not None
    with torch.inference_mode():
        assert same_bytes(ops.quantize_mxfp8(x, e).values, direct(x, e).values)
    half = calls["depthwise5x5_act"][0]
    assert same_bytes(ops.depthwise5x5_act(half[0].half(), *half[1:]), ops.depthwise5x5_act(half[0].half().to(BF16), *half[1:]))
    try:
        ops.configure("-quantize_mxfp8")
        with pytest.raises(ops.NoImplementation):
            ops.quantize_mxfp8(x, e)
    finally:
        ops.configure(None)


def test_native_calls_follow_the_current_stream(ops):
    (x, e), _ = _calls(ops)["quantize_mxfp8"]
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    ops.quantize_mxfp8(x, e)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        captured = ops.quantize_mxfp8(x, e).values
    captured.view(torch.uint8).zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert same_bytes(captured, ops.quantize_mxfp8(x, e).values)
