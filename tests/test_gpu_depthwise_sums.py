"""The depthwise kernel's sums against an fp32 chain: tap by tap from the first to the last, the bias at the end. The products of
two bf16 values are exact in fp32, so the chain of multiply-adds is a chain of products and sums."""

import pytest
import torch
import torch.nn.functional as F

from fim_testlib import DEV, bf16_ulp_distance, same_bytes

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    import flashim_b200

    yield flashim_b200.ops
    flashim_b200.ops.reset_call_counts()  # other modules count calls


@pytest.fixture(params=[0, 1], ids=["grid", "one-cta"])
def ctas(request):
    """One CTA: three quads walk every step of every channel tile, so that their lists fill many times over."""
    from flashim_b200 import _native

    _native.library().fim_dw_tune(request.param, 0)
    yield request.param
    _native.library().fim_dw_tune(0, 0)


def chain(x, w, b=None):
    """``x`` bf16 NHWC, ``w`` bf16 ``[25, C]`` -> fp32 NHWC."""
    height, width = x.shape[1:3]
    padded, total = F.pad(x.float(), (0, 0, 2, 2, 2, 2)), torch.zeros(x.shape, device=x.device)
    for tap in range(25):
        ky, kx = divmod(tap, 5)
        total = total + padded[:, ky: ky + height, kx: kx + width] * w[tap].float()
    return total if b is None else total + b


def cancelling(shape, seed, where):
    """Normal data with 5 x 5 areas of one value each around the pixels of ``where``, over which the bias cancels the sum up to
    the roundings: what is left there differs with the order of the sum."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    batch, height, width, c = shape
    x, w = torch.randn(shape, generator=g, device=DEV).to(BF16), torch.randn(25, c, generator=g, device=DEV).to(BF16)
    level = torch.randn(c, generator=g, device=DEV).to(BF16)
    flat = F.max_pool2d(where.float()[:, None], 5, 1, 2)[:, 0].bool()
    x = torch.where(flat[..., None], level, x)
    return x, w, -(w.double().sum(0) * level.double()).float()


@pytest.mark.parametrize("everywhere", [False, True], ids=["patches", "flat image"])
def test_no_cancelled_output_is_lost(ops, ctas, everywhere):
    """Every output listed for its cancellation comes out as the chain has it, however many there are: 32 channels of one
    pixel in some steps, whole steps, and lists that fill up on the way."""
    shape = (2, 49, 101, 96)
    where = torch.zeros(shape[:3], dtype=torch.bool, device=DEV)
    where[:, 4::8, 5::11] = True
    if everywhere:
        where[:] = True
    x, w, b = cancelling(shape, 5, where)
    want = chain(x, w, b).to(BF16)
    inner = where.clone()  # windows that the padding does not cut
    inner[:, :2], inner[:, -2:], inner[:, :, :2], inner[:, :, -2:] = False, False, False, False
    got = [ops.depthwise5x5_act(x.permute(0, 3, 1, 2), w, b, "none") for _ in range(3)]
    assert same_bytes(got[0][inner], want[inner])
    assert int(bf16_ulp_distance(got[0][~inner], want[~inner]).max() if not inner.all() else 0) <= 1
    assert same_bytes(got[1], got[0]) and same_bytes(got[2], got[0])


def test_what_is_not_finite_costs_its_own_steps(ops, ctas):
    """The patches (6 x 8 pixels) that hold an infinity are summed again with their step of 4 rows x 32 columns x 32 channels;
    every other step keeps the bytes that it has without the infinity, and the windows that hold it have the chain's."""
    shape = (2, 61, 130, 64)
    g = torch.Generator(device=DEV).manual_seed(3)
    x, w = torch.randn(shape, generator=g, device=DEV).to(BF16), (torch.randn(25, 64, generator=g, device=DEV) * 0.2).to(BF16)
    b = torch.randn(64, generator=g, device=DEV)
    spoiled, redone = x.clone(), torch.zeros(shape, dtype=torch.bool, device=DEV)
    for image, y, px, c, value in ((0, 0, 0, 3, float("inf")), (0, 30, 63, 40, float("nan")), (1, 60, 129, 63, float("-inf"))):
        spoiled[image, y, px, c] = value
        for top in range(0, shape[1], 4):
            for left in range(0, shape[2], 32):
                if top - 2 <= y <= top + 5 and left - 2 <= px <= left + 33:
                    redone[image, top: top + 4, left: left + 32, c // 32 * 32: c // 32 * 32 + 32] = True
    clean, got = (ops.depthwise5x5_act(t.permute(0, 3, 1, 2), w, b, "none") for t in (x, spoiled))
    assert same_bytes(got[~redone], clean[~redone])
    want = chain(spoiled, w, b).to(BF16)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    number = redone & ~torch.isnan(want)
    assert number.any() and same_bytes(got[number], want[number])
    assert int((~torch.isfinite(want)).sum()) > 0
