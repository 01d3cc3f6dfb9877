"""Spatial convs whose tiles take one halo patch of activations (narrow outputs, resident weights) against the schedule that
streams a shifted tile per tap (flag 2048): the same MMAs in the same order, hence the same bytes, and INT8 against the oracle."""

import pytest
import torch

import oracle
from fim_testlib import conv_schedule, same_bytes, to_dev

pytestmark = pytest.mark.gpu
E4M3, BF16 = torch.float8_e4m3fn, torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    import flashim_b200

    yield flashim_b200.ops
    flashim_b200.ops.reset_call_counts()  # other modules count calls


CASES = [  # batch, height, width, cin, cout, kh, kw, ph, pw, dh, dw, most CTAs
    (1, 16, 8, 64, 64, 3, 3, 1, 1, 1, 1, 0), (3, 17, 9, 64, 64, 3, 3, 1, 1, 1, 1, 2), (2, 33, 41, 128, 128, 3, 3, 1, 1, 1, 1, 5),
    (2, 31, 23, 32, 32, 5, 5, 2, 2, 1, 1, 3), (1, 20, 20, 96, 96, 3, 3, 2, 2, 2, 2, 1), (1, 1, 50, 64, 128, 1, 3, 0, 1, 1, 1, 2),
    (2, 12, 7, 128, 64, 3, 1, 0, 0, 3, 1, 0), (1, 6, 6, 64, 64, 3, 3, 0, 0, 1, 1, 0), (1, 40, 30, 192, 64, 3, 3, 1, 1, 1, 1, 4),
    (4, 40, 40, 64, 64, 3, 3, 1, 1, 1, 1, 1),  # tiles enough for several copies of the GELU table
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%dx%dx%d_c%d-%d_k%dx%d_p%d%d_d%d%d_ctas%d" % c)
def test_patches_equal_shifted_tiles(ops, case):
    b, h, w, cin, cout, kh, kw, ph, pw, dh, dw, ctas = case
    geometry = (kh, kw, 1, 1, ph, pw, dh, dw)
    g = torch.Generator().manual_seed(sum(case))
    bias = torch.randn(cout, generator=g).to(BF16)
    x, weight = (torch.randn(b, h, w, cin, generator=g) * 2).to(E4M3), torch.randn(cout, kh * kw * cin, generator=g).to(E4M3)
    ce = torch.randint(-5, 2, (cin // 32,), dtype=torch.int8, generator=g)
    we = torch.randint(-9, -3, (cout, kh * kw * cin // 32), dtype=torch.int8, generator=g)
    oe = torch.full((cout // 32,), -3, dtype=torch.int8)
    xi = torch.randint(-127, 128, (b, h, w, cin), dtype=torch.int8, generator=g)
    wi = torch.randint(-127, 128, (cout, kh * kw * cin), dtype=torch.int8, generator=g)
    ws, scale = torch.rand(cout, generator=g) * 1e-3, torch.tensor(0.02)
    mx = to_dev(x, ce, weight, oracle.swizzle_32_4_4(we), bias)
    i8 = to_dev(xi, wi, scale, ws, bias)

    def run():
        outs = [ops.mxfp8_conv2d_fused(*mx, *geometry), ops.mxfp8_conv2d_fused(*mx, *geometry, act="gelu", out_exponent=to_dev(oe)),
                ops.mxfp8_conv2d_fused(*mx, *geometry, out_fp32=True), *ops.mxfp8_conv2d_fused(*mx, *geometry, dynamic_out=True),
                ops.int8_conv2d(*i8, *geometry, relu=True)]
        if min(outs[0].shape[1:3]) >= 2:
            outs += ops.int8_conv2d_maxpool(*i8, *geometry, out_scale=to_dev(scale))
        return outs

    with conv_schedule(0, ctas, 2048):
        want = run()
    with conv_schedule(0, ctas):
        got = run()
    assert len(got) == len(want) and all(same_bytes(p, q) for p, q in zip(got, want))
    assert same_bytes(got[5].cpu(), oracle.int8_conv2d(xi, wi, scale, ws, bias, *geometry, relu=True))
