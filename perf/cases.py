"""Performance cases: the calls that programs built on this framework make, through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (device tensors, packed weights, a
loaded model), ``run`` is one pass. ``listed`` names the cases of a report, ``draw`` takes others from the same ranges.

Kinds:
  conv-mx    a static MXFP8 conv layer: activation quantiser (left out where the layer before hands over E4M3) + conv
  conv-int8  the same for INT8, optionally with the pooled second output of an encoder stage
  depthwise  the dense or INT8 depthwise 5x5 producer
  separable  a depthwise-separable refiner block in one of its three precisions
  linear     the static MXFP8 / INT8 linears and the GELU MLP of a transformer block
  glue       a RoMaV2 refiner step's first and last launch: input rows and warp / confidence heads
  stack      the refiner stack through ``load()``, eager or as a CUDA graph
"""

from __future__ import annotations

import math

import torch

import flashim_b200
from flashim_b200 import ops
from flashim_b200.quant import (
    QuantizedTensor, QuantizedWeight, calibrate_block32_exponent, swizzle_scales,
)
from flashim_b200.quant.tensor import int8_weight_from_conv

BF16, E4M3 = torch.bfloat16, torch.float8_e4m3fn


def listed() -> list[dict]:
    return [
        # a layer of a one-image stream: launch and host cost count as much as the kernel
        _conv("conv-mx 1x64x64x128 k3", "conv-mx", 1, 64, 64, 128, 128, source="fp32"),
        # a down-sampling residual layer with sizes that fit no tile
        _conv("conv-mx 3x75x101x96 s2 res", "conv-mx", 3, 75, 101, 96, 160, stride=2, act="relu", residual=True),
        # the coarse and the fine end of the conv sweep, inside a chain of quantised layers
        _conv("conv-mx 4x100x100x512 k3", "conv-mx", 4, 100, 100, 512, 512, act="gelu", requant=True, source="codes"),
        _conv("conv-mx 4x800x800x64 k3", "conv-mx", 4, 800, 800, 64, 64, act="gelu", requant=True, source="codes"),
        # an INT8 layer fed by a chained one, and the last layer of an encoder stage with its pooled output
        _conv("conv-int8 2x100x100x256 k3", "conv-int8", 2, 100, 100, 256, 256, source="codes"),
        _conv("conv-int8 pool 4x201x199x128", "conv-int8", 4, 201, 199, 128, 128, act="relu", pool=True),
        # the memory-bound producer at its benchmark size
        {"name": "depthwise 4x200x200x256 gelu", "kind": "depthwise", "batch": 4, "height": 200, "width": 200, "cin": 256,
         "act": "gelu", "out": "bf16"},
        # one refiner block of a small, ragged image pair
        {"name": "separable mx 2x101x133x128", "kind": "separable", "batch": 2, "height": 101, "width": 133, "cin": 128,
         "precision": "mxfp8"},
        # a transformer MLP over one image's tokens
        {"name": "linear mlp 1000x256x1024", "kind": "linear", "form": "mlp", "rows": 1000, "cin": 256, "cout": 1024},
        # first and last launch of a refinement step, both directions of one pair
        {"name": "glue 2x96x72x64 r3", "kind": "glue", "batch": 2, "height": 96, "width": 72, "features": 64, "channels": 128,
         "radius": 3},
        # one image pair called eagerly, and a batch of pairs as the benchmark serves it
        {"name": "stack eager 1 pair", "kind": "stack", "pairs": 1, "size": 50, "engine": "eager"},
        {"name": "stack graph 8 pairs", "kind": "stack", "pairs": 8, "size": 100, "engine": "cuda-graph"},
    ]


def _conv(name, kind, batch, height, width, cin, cout, k=3, stride=1, act="none", residual=False, requant=False, pool=False,
          source="bf16"):
    case = {"kind": kind, "batch": batch, "height": height, "width": width, "cin": cin, "cout": cout, "k": k, "stride": stride,
            "act": act, "residual": residual, "requant": requant, "pool": pool, "source": source}
    return case if name is None else {"name": name, **case}


# ---- drawn cases -------------------------------------------------------------------------------------------------------


def _log(rng, low, high) -> int:
    return round(math.exp(rng.uniform(math.log(low), math.log(high))))


def _image(rng, channels, most, high=800):
    """Batch, height and width, any remainders, of at most ``most`` elements."""
    while True:
        batch, height, width = rng.randint(1, 4), _log(rng, 16, high), 0
        width = max(5, min(high, round(height * rng.uniform(0.6, 1.6))))
        if batch * height * width * channels <= most:
            return batch, height, width


def draw(rng) -> dict:
    kind = rng.choice(["conv-mx", "conv-mx", "conv-mx", "conv-int8", "conv-int8", "depthwise", "separable", "linear", "glue", "stack"])
    if kind in ("conv-mx", "conv-int8"):
        cin = rng.choice([32, 64, 64, 96, 128, 128, 192, 256, 512])
        cout = rng.choice([cin, cin, cin, min(512, 2 * cin), 160])
        batch, height, width = _image(rng, max(cin, cout), 80_000_000)
        k, stride = rng.choice([3, 3, 3, 1]), rng.choice([1, 1, 1, 2])
        source, act = rng.choice(["bf16", "codes"]), rng.choice(["none", "relu"])
        if kind == "conv-int8":
            pool = rng.random() < 0.3
            return _conv(None, kind, batch, height, width, cin, cout, k, stride, act, residual=not pool and rng.random() < 0.3,
                         pool=pool, requant=not pool and rng.random() < 0.3, source=source)
        if rng.random() < 0.3:
            act = "gelu"
        return _conv(None, kind, batch, height, width, cin, cout, k, stride, act, residual=rng.random() < 0.3,
                     requant=rng.random() < 0.4, source=rng.choice([source, "fp32"]))
    if kind == "depthwise":
        cin = rng.choice([32, 64, 128, 256, 512])
        batch, height, width = _image(rng, cin, 80_000_000, 400)
        out = rng.choice(["bf16", "bf16", "int8"])
        return {"kind": kind, "batch": batch, "height": height, "width": width, "cin": cin,
                "act": "relu" if out == "int8" else rng.choice(["gelu", "relu"]), "out": out}
    if kind == "separable":
        cin = rng.choice([32, 128, 128, 512])
        batch, height, width = _image(rng, cin, 40_000_000, 400)
        return {"kind": kind, "batch": batch, "height": height, "width": width, "cin": cin,
                "precision": rng.choice(["bf16", "mxfp8", "int8"])}
    if kind == "linear":
        cin = rng.choice([128, 256, 384, 768, 1024])
        return {"kind": kind, "form": rng.choice(["mlp", "mxfp8", "int8"]), "rows": _log(rng, 16, 20000), "cin": cin, "cout": 4 * cin}
    if kind == "glue":
        features = rng.choice([32, 64, 128])
        batch, height, width = _image(rng, features, 10_000_000, 320)
        return {"kind": kind, "batch": 2 * ((batch + 1) // 2), "height": height, "width": width, "features": features,
                "channels": rng.choice([32, 128, 512]), "radius": rng.choice([2, 3])}
    pairs, size = rng.randint(1, 8), _log(rng, 20, 60)
    return {"kind": "stack", "pairs": pairs, "size": size, "engine": rng.choice(["eager", "cuda-graph"])}


# ---- inputs ------------------------------------------------------------------------------------------------------------


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(dtype)


def prepare(case: dict, seed: int) -> dict:
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {"case": case, **_PREPARE[case["kind"]](case, g)}


def _out(size: int, k: int, stride: int) -> int:
    return (size + 2 * (k // 2) - k) // stride + 1


def _prepare_conv(case, g):
    b, h, w, cin, cout, k, stride = (case[n] for n in ("batch", "height", "width", "cin", "cout", "k", "stride"))
    x = _randn(g, b, h, w, cin, dtype=torch.float32 if case["source"] == "fp32" else BF16)
    weight = _randn(g, cout, cin, k, k, scale=math.sqrt(2 / (cin * k * k)))
    state = {"geometry": (k, k, stride, stride, k // 2, k // 2, 1, 1), "bias": _randn(g, cout, scale=0.02, dtype=BF16), "residual": None}
    if case["residual"]:
        state["residual"] = _randn(g, b, _out(h, k, stride), _out(w, k, stride), cout, dtype=BF16)
    if case["kind"] == "conv-mx":
        packed = QuantizedWeight.from_conv(weight)
        exponent = calibrate_block32_exponent(x)
        state.update(exponent=exponent, weight=packed.values, weight_exponent=packed.scale_exponent,
                     weight_scales=swizzle_scales(packed.scale_exponent))
        # activations of unit variance leave the layer with a variance near 2: +-16 covers them
        state["out_exponent"] = torch.full((cout // 32,), -4, dtype=torch.int8, device="cuda") if case["requant"] else None
        state["x"] = ops.quantize_mxfp8(x, exponent).values if case["source"] == "codes" else x
    else:
        codes, scales = int8_weight_from_conv(weight)
        state.update(weight=codes, weight_scale=scales, scale=x.abs().amax().float() / 127)
        state["out_scale"] = torch.tensor(8 / 127, device="cuda") if case["requant"] or case["pool"] else None
        state["x"] = ops.quantize_int8(x, state["scale"]).values if case["source"] == "codes" else x
    return state


def _prepare_depthwise(case, g):
    b, h, w, c = (case[n] for n in ("batch", "height", "width", "cin"))
    return {"x": _randn(g, b, h, w, c, dtype=BF16).permute(0, 3, 1, 2), "weight": _randn(g, 25, c, scale=0.05, dtype=BF16),
            "bias": _randn(g, c, scale=0.02), "scale": torch.tensor(0.01, device="cuda")}


def _prepare_separable(case, g):
    c, state = case["cin"], _prepare_depthwise(case, g)
    pointwise = _randn(g, c, c, 1, 1, scale=math.sqrt(2 / c))
    state["pw_bias"] = _randn(g, c, scale=0.02, dtype=BF16)
    if case["precision"] == "bf16":
        state["pw"] = pointwise.reshape(c, c).to(BF16)
    elif case["precision"] == "mxfp8":
        packed = QuantizedWeight.from_conv(pointwise)
        state.update(pw=packed.values, pw_swizzled=swizzle_scales(packed.scale_exponent).view(torch.float8_e8m0fnu),
                     pw_plain=(packed.scale_exponent.int() + 127).to(torch.uint8))
    else:
        state["pw"], state["pw_scale"] = int8_weight_from_conv(pointwise)
    return state


def _prepare_linear(case, g):
    rows, cin, cout = case["rows"], case["cin"], case["cout"]
    x = _randn(g, rows, cin, dtype=BF16)
    weight = _randn(g, cout, cin, scale=math.sqrt(1 / cin))
    if case["form"] == "int8":
        codes, scales = int8_weight_from_conv(weight.reshape(cout, cin, 1, 1))
        return {"x": x, "scale": x.abs().amax().float() / 127, "weight": codes, "weight_scale": scales,
                "bias": _randn(g, cout, scale=0.02, dtype=BF16), "residual": _randn(g, rows, cout, dtype=BF16)}
    return {"x": x, "exponent": calibrate_block32_exponent(x), "w1": QuantizedWeight.from_float(weight),
            "bias": _randn(g, cout, scale=0.02, dtype=BF16),
            "hidden": torch.full((cout // 32,), -6, dtype=torch.int8, device="cuda"),
            "w2": QuantizedWeight.from_float(_randn(g, cin, cout, scale=math.sqrt(1 / cout))) if case["form"] == "mlp" else None}


def _prepare_glue(case, g):
    b, h, w, p, c = (case[n] for n in ("batch", "height", "width", "features", "channels"))
    gy, gx = torch.meshgrid(torch.linspace(-1 + 1 / h, 1 - 1 / h, h, device="cuda"), torch.linspace(-1 + 1 / w, 1 - 1 / w, w, device="cuda"),
                            indexing="ij")
    # a smooth displacement of some pixels plus noise, as a coarse match gives
    shift = torch.stack((torch.sin(3 * gy), torch.cos(2 * gx)), -1) * 0.1
    warp = torch.stack((gx, gy), -1) + shift + _randn(g, b, h, w, 2, scale=0.01)
    features = _randn(g, b, h, w, p)
    return {"features": features, "warp": warp.contiguous(), "emb_weight": _randn(g, 32, 2), "emb_bias": _randn(g, 32),
            "scale": (3.0, 2.0), "z": _randn(g, b, h, w, c, dtype=BF16).permute(0, 3, 1, 2),
            "head": _randn(g, 6, c, scale=0.1), "head_bias": _randn(g, 6), "confidence": _randn(g, b, h, w, 4)}


def _stack_levels(case):
    return ((case["size"], 512), (2 * case["size"], 256), (4 * case["size"], 128))


def _prepare_stack(case, g):
    levels = _stack_levels(case)
    model = flashim_b200.load("refiner-stack", "fp8", device="cuda", engine=case["engine"],
                              overrides={"arch.levels": [list(level) for level in levels]})
    return {"model": model, "pyramid": [_randn(g, 2 * case["pairs"], s, s, c, dtype=BF16) for s, c in levels]}


_PREPARE = {"conv-mx": _prepare_conv, "conv-int8": _prepare_conv, "depthwise": _prepare_depthwise, "separable": _prepare_separable,
            "linear": _prepare_linear, "glue": _prepare_glue, "stack": _prepare_stack}


# ---- one pass ----------------------------------------------------------------------------------------------------------


def run(state: dict):
    return _RUN[state["case"]["kind"]](state["case"], state)


def _run_conv_mx(case, s):
    x = s["x"] if case["source"] == "codes" else ops.quantize_mxfp8(s["x"], s["exponent"]).values
    if case["act"] == "gelu":
        return ops.mxfp8_conv2d_fused(x, s["exponent"], s["weight"], s["weight_scales"], s["bias"], *s["geometry"], act="gelu",
                                      residual=s["residual"], out_exponent=s["out_exponent"])
    return ops.mxfp8_conv2d(x, s["exponent"], s["weight"], s["weight_exponent"], s["bias"], *s["geometry"],
                            relu=case["act"] == "relu", residual=s["residual"], out_exponent=s["out_exponent"])


def _run_conv_int8(case, s):
    x = s["x"] if case["source"] == "codes" else ops.quantize_int8(s["x"], s["scale"]).values
    if case["pool"]:
        return ops.int8_conv2d_maxpool(x, s["weight"], s["scale"], s["weight_scale"], s["bias"], *s["geometry"],
                                       relu=case["act"] == "relu", out_scale=s["out_scale"])
    return ops.int8_conv2d(x, s["weight"], s["scale"], s["weight_scale"], s["bias"], *s["geometry"], relu=case["act"] == "relu",
                           residual=s["residual"], out_scale=s["out_scale"])


def _run_depthwise(case, s):
    if case["out"] == "int8":
        return ops.depthwise5x5_relu_int8(s["x"], s["weight"], s["bias"], s["scale"])
    return ops.depthwise5x5_act(s["x"], s["weight"], s["bias"], case["act"])


def _run_separable(case, s):
    if case["precision"] == "bf16":
        return ops.depthwise5x5_relu_pointwise(s["x"], s["weight"], s["bias"], s["pw"], s["pw_bias"])
    if case["precision"] == "mxfp8":
        return ops.depthwise5x5_relu_pointwise_mxfp8(s["x"], s["weight"], s["bias"], s["pw"], s["pw_swizzled"], s["pw_plain"], s["pw_bias"])
    return ops.depthwise5x5_relu_pointwise_int8(s["x"], s["weight"], s["bias"], s["pw"], s["pw_scale"], s["pw_bias"], s["scale"])


def _run_linear(case, s):
    if case["form"] == "int8":
        x = ops.quantize_int8(s["x"], s["scale"])
        return ops.int8_linear(x.values, s["weight"], x.scale, s["weight_scale"], s["bias"], gelu=True, residual=s["residual"])
    x: QuantizedTensor = ops.quantize_mxfp8(s["x"], s["exponent"])
    if case["form"] == "mxfp8":
        return ops.mxfp8_linear(x, s["bias"], s["w1"])
    return ops.mxfp8_gelu_mlp(x, s["w1"], s["bias"], s["hidden"], s["w2"])


def _run_glue(case, s):
    rows = ops.romav2_refiner_input(s["features"], s["features"], s["warp"], s["emb_weight"], s["emb_bias"], s["scale"],
                                    case["radius"], case["batch"] // 2)
    return rows, ops.romav2_refiner_heads(s["z"], s["head"], s["head_bias"], s["warp"], s["confidence"], 4.0)


def _run_stack(case, s):
    return s["model"](s["pyramid"])


_RUN = {"conv-mx": _run_conv_mx, "conv-int8": _run_conv_int8, "depthwise": _run_depthwise, "separable": _run_separable,
        "linear": _run_linear, "glue": _run_glue, "stack": _run_stack}


# ---- what a pass cannot do without, and how near another implementation comes ---------------------------------------------


def work(case: dict) -> dict:
    """Bytes of every input and output once, and the operations of the arithmetic itself."""
    kind = case["kind"]
    if kind in ("conv-mx", "conv-int8"):
        b, h, w, cin, cout, k, stride = (case[n] for n in ("batch", "height", "width", "cin", "cout", "k", "stride"))
        pixels = b * _out(h, k, stride) * _out(w, k, stride)
        read = b * h * w * cin * {"codes": 1, "bf16": 2, "fp32": 4}[case["source"]] + cout * k * k * cin * 33 / 32
        write = pixels * cout * (1 if case["requant"] else 2) + (pixels // 4 * cout if case["pool"] else 0)
        return {"bytes": read + write + (2 * pixels * cout if case["residual"] else 0), "flops": 2 * pixels * cout * cin * k * k}
    if kind in ("depthwise", "separable"):
        elements = case["batch"] * case["height"] * case["width"] * case["cin"]
        if kind == "depthwise":
            return {"bytes": elements * (2 + (1 if case["out"] == "int8" else 2)), "flops": 50 * elements}
        return {"bytes": 4 * elements, "flops": (50 + 2 * case["cin"]) * elements}
    if kind == "linear":
        rows, cin, cout = case["rows"], case["cin"], case["cout"]
        products, weights = (2, 2 * cin * cout) if case["form"] == "mlp" else (1, cin * cout)
        out = 2 * rows * (cin if case["form"] == "mlp" else cout)
        return {"bytes": 2 * rows * cin + weights + out * (2 if case["form"] == "int8" else 1), "flops": 2 * products * rows * cin * cout}
    if kind == "glue":
        pixels, p, k = case["batch"] * case["height"] * case["width"], case["features"], (2 * case["radius"] + 1) ** 2
        return {"bytes": pixels * (4 * p + 8 + 2 * (2 * p + 32 + k) + 2 * case["channels"] + 8 + 16 + 8 + 16),
                "flops": pixels * (2 * p * (2 * case["radius"] + 2) ** 2 + 8 * p + 12 * case["channels"])}
    images, total, flops = 2 * case["pairs"], 0, 0
    for size, c in _stack_levels(case):
        pixels = images * size * size
        total += pixels * (2 * c + 2 * 32)
        flops += pixels * (2 * c * c + 4 * (50 * c + 8 * c * c) + 2 * c * 4)
    return {"bytes": total, "flops": flops}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "conv-int8":
        return "exact"  # integer sums, one fixed order of roundings after them
    if kind == "conv-mx":
        # fp32 sums in another order: a bf16 result may land one ulp away, and an E4M3 code made from it one code (2**-3)
        return {"rel": 4e-3, "max": 0.13} if case["requant"] else {"rel": 2e-3, "max": 0.02}
    if kind == "depthwise":
        return {"rel": 0.0, "differ": 1e-3} if case["out"] == "int8" else {"rel": 2e-3, "max": 0.01}
    if kind == "separable":
        return {"rel": 4e-3, "max": 0.1}  # a hidden code that flips moves an output by its quantum
    if kind == "linear":
        return "exact" if case["form"] == "int8" else {"rel": 5e-3, "max": 0.1}
    if kind == "glue":
        return {"rel": 2e-3, "max": 0.02}
    return {"rel": 1e-2, "max": 0.3}  # six quantisers in a row, each may flip one code in a thousand
