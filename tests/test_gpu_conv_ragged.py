"""Convs whose input channels 128 does not divide, in 128-byte K steps with a short last one per tap, against the steps that divide
them (flag 32768): the same products in the same order, hence the same bytes, and INT8 against the oracle."""

import ctypes

import pytest
import torch

import oracle
from fim_testlib import conv_schedule, same_bytes, to_dev

E4M3, BF16 = torch.float8_e4m3fn, torch.bfloat16
CASES = [  # batch, height, width, cin, cout, kernel, stride, padding, dilation, most CTAs, forced tile width
    (3, 38, 51, 96, 160, 3, 2, 1, 1, 0, 0), (1, 17, 9, 160, 128, 3, 1, 1, 1, 2, 0), (2, 20, 23, 192, 192, 3, 1, 1, 1, 3, 0),
    (1, 19, 21, 96, 96, 3, 1, 1, 1, 2, 0), (1, 19, 21, 96, 64, 3, 1, 2, 2, 1, 0), (1, 30, 20, 224, 64, 1, 1, 0, 1, 2, 0),
    (2, 13, 13, 480, 256, 3, 1, 1, 1, 2, 128), (1, 40, 45, 288, 512, 1, 1, 0, 1, 5, 128), (1, 15, 14, 96, 32, 5, 3, 2, 1, 0, 0),
    (1, 16, 16, 672, 128, 3, 1, 1, 1, 0, 0), (1, 129, 1, 96, 288, 1, 1, 0, 1, 1, 0), (1, 5, 5, 1120, 64, 3, 1, 1, 1, 0, 0),
    # tiles of 256 columns, made narrower for few of them
    (1, 40, 40, 192, 256, 3, 1, 1, 1, 0, 0), (1, 21, 19, 160, 512, 3, 2, 1, 1, 0, 0), (1, 40, 40, 96, 256, 1, 1, 0, 1, 0, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%dx%dx%d_c%d-%d_k%d_s%d_p%d_d%d_ctas%d_n%d" % c)
def test_ragged_steps_equal_divided_steps(case):
    import flashim_b200

    ops = flashim_b200.ops
    b, h, w, cin, cout, k, stride, pad, dil, ctas, width = case
    geometry = (k, k, stride, stride, pad, pad, dil, dil)
    g = torch.Generator().manual_seed(sum(case))
    bias = torch.randn(cout, generator=g).to(BF16)
    x, weight = (torch.randn(b, h, w, cin, generator=g) * 2).to(E4M3), torch.randn(cout, k * k * cin, generator=g).to(E4M3)
    ce = torch.randint(-5, 2, (cin // 32,), dtype=torch.int8, generator=g)
    we = torch.randint(-9, -3, (cout, k * k * cin // 32), dtype=torch.int8, generator=g)
    oe = torch.full((cout // 32,), -3, dtype=torch.int8)
    xi = torch.randint(-127, 128, (b, h, w, cin), dtype=torch.int8, generator=g)
    wi = torch.randint(-127, 128, (cout, k * k * cin), dtype=torch.int8, generator=g)
    ws, scale = torch.rand(cout, generator=g) * 1e-3, torch.tensor(0.02)
    mx, i8 = to_dev(x, ce, weight, oracle.swizzle_32_4_4(we), bias), to_dev(xi, wi, scale, ws, bias)

    def run():
        plain = ops.mxfp8_conv2d_fused(*mx, *geometry)
        return [plain, ops.mxfp8_conv2d_fused(*mx, *geometry, act="gelu", out_exponent=to_dev(oe)),
                ops.mxfp8_conv2d_fused(*mx, *geometry, residual=plain, out_fp32=False), *ops.mxfp8_conv2d_fused(*mx, *geometry, act="gelu", dynamic_out=True),
                ops.int8_conv2d(*i8, *geometry, relu=True), ops.int8_conv2d_accumulators(*i8[:2], *geometry)]

    with conv_schedule(width, ctas, 32768):
        want = run()
    with conv_schedule(width, ctas):
        got = run()
    assert all(same_bytes(p, q) for p, q in zip(got, want, strict=True))
    assert same_bytes(got[5].cpu(), oracle.int8_conv2d(xi, wi, scale, ws, bias, *geometry, relu=True))
    flashim_b200.ops.reset_call_counts()  # other modules count calls


def test_plans_take_ragged_steps_where_they_serve():
    """Widths of the tiles and of their K steps: 128 bytes for channels that 64 does not divide, or 64 does (MXFP8 alone); not for two blocks or
    fewer, nor for tiles that are 256 wide in the end."""
    from flashim_b200 import _native

    lib = _native.library()

    def plan(cin, int8, k=3, cout=160, size=40):
        geometry = _native.ConvGeometry(1, size, size, cin, cout, k, k, 1, 1, k // 2, k // 2, 1, 1)
        plan = (ctypes.c_int * 6)()
        assert lib.fim_conv_plan(ctypes.byref(geometry), int8, 0, ctypes.byref(plan)) == 0
        return plan[2], plan[3]

    def step(*args, **kw):
        return plan(*args, **kw)[1]

    assert [step(c, 0) for c in (32, 64, 96, 128, 160, 192)] == [32, 64, 128, 128, 128, 128]
    assert [step(c, 1) for c in (32, 64, 96, 128, 160, 192)] == [32, 64, 128, 128, 128, 64]
    assert step(992, 0) == 32 and step(992, 0, k=1) == 128  # weight scales of nine taps: more than tensor memory holds
    assert step(192, 0, cout=64) == 64  # keeps its halo patches
    # a 256-wide tile, and one that few tiles make narrower
    assert plan(192, 0, cout=256, size=200) == (256, 64) and plan(192, 0, cout=256) == (128, 128) and plan(192, 0, cout=512, size=50) == (128, 128)
    assert plan(96, 0, k=1, cout=256, size=200) == (256, 32) and plan(96, 0, k=1, cout=256) == (128, 128)
    assert plan(160, 1, cout=256, size=200) == (256, 32) and plan(160, 1, cout=256, size=20) == (64, 128)
    # patches: while a CTA has few of them to walk, up to six
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
    for size in (72, 136, 200, 240, 264, 400):  # 8 x 16 pixels each
        tiles = -(-size // 8) * -(-size // 16)
        assert step(96, 0, cout=64, size=size) == (128 if tiles <= 6 * min(sms, tiles) else 32)
    # the kernel has no CTA pairs with ragged steps: none are planned, whatever is asked for
    for cin, int8, size, k in ((96, 0, 400, 3), (160, 0, 200, 1), (96, 1, 200, 3), (160, 1, 400, 1)):
        for flags in (0, 128, 16384, 128 | 16384):
            for width in (0, 128, 256):
                with conv_schedule(width, 0, flags) as c:
                    ragged = plan(cin, int8, k, 512, size)[1] == 128
                    assert not (ragged and c.schedule((1, size, size, cin, 512, k, k, k // 2, 1), bool(int8))["pairs"])
                    assert ragged or width != 128
