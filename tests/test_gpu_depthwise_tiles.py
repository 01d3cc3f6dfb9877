"""The depthwise kernel at the edges of its tiles: 32 columns x 4 rows x 32 channels per step, quads of warps that walk
several spans and channel tiles when the grid is small, outputs that TMA cannot store to."""

import pytest
import torch

import oracle
from fim_testlib import DEV, bf16_ulp_distance, code_mismatch, same_bytes, to_dev

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    import flashim_b200

    yield flashim_b200.ops
    flashim_b200.ops.reset_call_counts()  # other modules count calls


@pytest.mark.parametrize("ctas", [0, 1])
@pytest.mark.parametrize("shape", [(1, 32, 1, 31), (2, 96, 4, 32), (1, 160, 5, 33), (1, 64, 3, 65), (2, 480, 8, 1), (1, 1056, 9, 40)])
def test_tile_edges(ops, shape, ctas):
    from flashim_b200 import _native

    g = torch.Generator().manual_seed(sum(shape))
    x = torch.randn(shape, generator=g).to(BF16).contiguous(memory_format=torch.channels_last)
    w, b = (torch.randn(25, shape[1], generator=g) * 0.2).to(BF16), torch.randn(shape[1], generator=g)
    xd, wd, bd = to_dev(x, w, b)
    lib = _native.library()
    try:
        lib.fim_dw_tune(ctas, 0)  # one CTA: three quads walk every span of every channel tile
        dense = ops.depthwise5x5_act(xd, wd, bd, "relu")
        q, s = ops.depthwise5x5_relu_mxfp8(xd, wd, bd)
        codes = ops.depthwise5x5_relu_int8(xd, wd, bd, torch.tensor(0.03, device=DEV))
    finally:
        lib.fim_dw_tune(0, 0)
    assert int(bf16_ulp_distance(dense.cpu(), oracle.depthwise5x5_act_ext(x, w, b, "relu")).max()) <= 1
    q_ref, s_ref = oracle.depthwise5x5_relu_mxfp8(x, w, b)
    assert code_mismatch(q, q_ref) < 1e-3 and float((s.cpu().view(torch.uint8) != s_ref).float().mean()) < 1e-4
    want = oracle.depthwise5x5_relu_int8(x, w, b, torch.tensor(0.03))
    assert float((codes.cpu() != want).float().mean()) < 5e-3 and int((codes.cpu().int() - want.int()).abs().max()) <= 1


def test_tensor_core_sums_are_as_exact_as_an_fp32_chain(ops):
    """Against fp64, through the dense output without bias and activation: no more than twice as many outputs as of the fp32 chain
    are rounded to the wrong side of a bf16 boundary."""
    g = torch.Generator().manual_seed(1)
    x = torch.randn(1, 64, 40, 50, generator=g).to(BF16).contiguous(memory_format=torch.channels_last)
    w, b = torch.randn(25, 64, generator=g).to(BF16), torch.zeros(64)
    dense = ops.depthwise5x5_act(*to_dev(x, w, b), "none").cpu()
    kernel = w.double().t().reshape(64, 1, 5, 5)
    exact = torch.nn.functional.conv2d(x.double(), kernel, padding=2, groups=64).permute(0, 2, 3, 1)
    chain = oracle.depthwise5x5_fp32(x, w, b).permute(0, 2, 3, 1)
    wrong = lambda v: float((v.to(BF16) != exact.to(BF16)).float().mean())  # noqa: E731  roundings on the wrong side
    assert wrong(dense) <= 2 * wrong(chain) + 2e-5


@pytest.mark.parametrize("offset", [4, 16])
def test_outputs_off_the_tma_alignment(offset):
    from flashim_b200 import _native

    b, h, w, c = 1, 6, 35, 64
    g = torch.Generator().manual_seed(2)
    x, wt, bias = torch.randn(b, h, w, c, generator=g).to(BF16).to(DEV), torch.randn(25, c, generator=g).to(BF16).to(DEV), torch.randn(c, generator=g).to(DEV)
    n = b * h * w * c
    lib, stream = _native.library(), torch.cuda.current_stream().cuda_stream
    outs = []
    for at in (0, offset):
        space = torch.full((4 * n + 64,), 7, dtype=torch.uint8, device=DEV)
        dense, codes = space[at: at + 2 * n], space[2 * n + 32 + at: 3 * n + 32 + at]
        scales = torch.zeros(b * h * w * (c // 32), dtype=torch.uint8, device=DEV)
        assert lib.fim_dw5x5_bf16(x.data_ptr(), wt.data_ptr(), bias.data_ptr(), dense.data_ptr(), b, h, w, c, 2, None, stream) == 0
        assert lib.fim_dw5x5_mxfp8(x.data_ptr(), wt.data_ptr(), bias.data_ptr(), codes.data_ptr(), scales.data_ptr(), 0, b, h, w, c, 2, None, stream) == 0
        torch.cuda.synchronize()
        assert int(space[3 * n + 32 + at]) == 7 and int(space[2 * n + at]) == 7  # nothing behind the outputs
        outs.append((dense.clone(), codes.clone(), scales))
    assert all(same_bytes(p, q) for p, q in zip(*outs))


def test_infinite_and_nan_inputs_stay_in_their_windows(ops):
    """The kernel multiplies a 6 x 8 patch per eight pixels; what is not finite may only show in the 5x5 windows that hold it."""
    g = torch.Generator().manual_seed(3)
    x = torch.randn(2, 64, 21, 70, generator=g).to(BF16).contiguous(memory_format=torch.channels_last)
    w, b = (torch.randn(25, 64, generator=g) * 0.2).to(BF16), torch.randn(64, generator=g)
    spoiled = x.clone(memory_format=torch.preserve_format)
    hit = torch.zeros(2, 21, 70, dtype=torch.bool)
    for image, c, y, px, v in ((0, 3, 0, 0, float("inf")), (0, 40, 10, 33, float("nan")), (1, 63, 20, 69, float("-inf")), (1, 0, 7, 31, float("nan"))):
        spoiled[image, c, y, px] = v
        hit[image, max(0, y - 2): y + 3, max(0, px - 2): px + 3] = True
    xd, sd, wd, bd = to_dev(x, spoiled, w, b)
    got, want = ops.depthwise5x5_act(sd, wd, bd, "none").cpu(), oracle.depthwise5x5_act_ext(spoiled, w, b, "none")
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[~finite & ~torch.isnan(want)], want[~finite & ~torch.isnan(want)])
    assert int(bf16_ulp_distance(got[finite], want[finite]).max()) <= 1
    scale = torch.tensor(0.03, device=DEV)
    for op, extra in ((ops.depthwise5x5_relu_int8, (scale,)), (lambda *a: ops.depthwise5x5_relu_mxfp8(*a)[0], ())):
        bad, clean = (op(t, wd, bd, *extra).cpu().view(torch.uint8).view(2, 21, 70, 64) for t in (sd, xd))
        assert float((bad[~hit] != clean[~hit]).float().mean()) < 1e-3
