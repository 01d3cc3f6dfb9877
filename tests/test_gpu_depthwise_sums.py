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


# ---- MXFP8: codes and scales of the chain ------------------------------------------------------------------------------

ACTS = {"none": 0, "relu": 1, "gelu": 2}


def quantise(values, act):
    """E4M3 codes ``[rows, C]`` and E8M0 bytes ``[rows, C / 32]`` of fp32 pre-activation values, by the op's own activation and
    quantiser: its sums over an image of zeros are zero in every order, so the bias of a channel passes through as it is."""
    from flashim_b200 import _native

    lib, rows, c = _native.library(), values.shape[0], values.shape[1]
    flat, step = values.reshape(-1).contiguous(), 1 << 20
    codes, scales = torch.empty(flat.numel(), dtype=torch.uint8, device=DEV), torch.empty(flat.numel() // 32, dtype=torch.uint8, device=DEV)
    x, w = torch.zeros(step, dtype=BF16, device=DEV), torch.zeros(25 * step, dtype=BF16, device=DEV)
    for at in range(0, flat.numel(), step):
        n = min(step, flat.numel() - at)
        part_codes, part_scales = torch.empty(n, dtype=torch.uint8, device=DEV), torch.empty(n // 32, dtype=torch.uint8, device=DEV)
        bias = flat[at: at + n].clone()
        assert lib.fim_dw5x5_mxfp8(x.data_ptr(), w.data_ptr(), bias.data_ptr(), part_codes.data_ptr(), part_scales.data_ptr(), 0, 1, 1, 1, n,
                                   ACTS[act], None, torch.cuda.current_stream().cuda_stream) == 0
        codes[at: at + n], scales[at // 32: (at + n) // 32] = part_codes, part_scales
    return codes.view(rows, c), scales.view(rows, c // 32)


def dw_mxfp8(x, w, b, act):
    from flashim_b200 import _native

    batch, height, width, c = x.shape
    rows = batch * height * width
    codes, scales = torch.empty(rows, c, dtype=torch.uint8, device=DEV), torch.empty(rows, c // 32, dtype=torch.uint8, device=DEV)
    assert _native.library().fim_dw5x5_mxfp8(x.data_ptr(), w.data_ptr(), b.data_ptr(), codes.data_ptr(), scales.data_ptr(), 0, batch, height, width, c,
                                             ACTS[act], None, torch.cuda.current_stream().cuda_stream) == 0
    return codes, scales


def data(kind, shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    batch, height, width, c = shape
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    x, w, b = rand(*shape), rand(25, c) * 0.05, rand(c) * 0.02
    zero_sum = rand(25, c) * 0.05
    zero_sum = (zero_sum - zero_sum.mean(0)).to(BF16).float()
    zero_sum[24] -= zero_sum.sum(0)  # (up to the rounding of one tap)
    if kind == "wide":  # arguments of the GELU of +-20: half of them in its tail
        w = w * 20
    elif kind == "smooth":
        x, w, b = F.interpolate(rand(batch, c, height // 8, width // 8), size=(height, width), mode="bicubic").permute(0, 2, 3, 1) + 10, zero_sum, b * 0
    elif kind == "edges":  # partial sums that grow over two rows of taps and shrink over the others
        x = F.interpolate(rand(batch, c, height // 8, width // 8), size=(height, width), mode="bicubic").permute(0, 2, 3, 1) + 3
        amplitude = torch.rand(5, 1, c, generator=g, device=DEV) * torch.tensor([1.0, 1.0, 0.0, -1.0, -1.0], device=DEV)[:, None, None]
        w, b = (amplitude.expand(5, 5, c) + 0.02 * rand(5, 5, c)).reshape(25, c), b * 0
    elif kind == "underflow":  # flat, with arguments at -12.743085, where the GELU goes from below zero to +0
        x, w, channel = rand(1, 1, 1, c).expand(shape).to(BF16), (rand(25, c) * 8).to(BF16), torch.arange(c, device=DEV)
        at = torch.where(channel % 32 == 5, 3.0, -12.743084 + (channel % 9 - 4) * 1e-6)
        b = (at - (x[0, 0, 0].double() * w.double()).sum(0)).float()
    elif kind == "flat":  # the sum of every window inside is what the roundings leave of zero
        x, w, b = rand(batch, 1, 1, c).expand(shape), zero_sum, b * 0
    elif kind == "heavy":
        x, w = (2 * x).exp() * rand(*shape).sign(), (2 * rand(25, c)).exp() * rand(25, c).sign()
    elif kind == "sparse":
        x = torch.where(F.avg_pool2d(rand(batch, 1, height, width), 9, 1, 4).permute(0, 2, 3, 1) > 0, x.relu(), 0.0)
    elif kind == "tiny":
        # (products of 2**-112 and down to 2**-133, below which 16 bits no longer fit and the product of the chain here would round)
        x, w, b = x * 1e-18, w * 1e-16, b * 0
    return x.to(BF16).contiguous(), w.to(BF16), b


@pytest.mark.parametrize("act", ["gelu", "relu", "none"])
@pytest.mark.parametrize("kind", ["normal", "wide", "smooth", "edges", "underflow", "flat", "heavy", "sparse", "tiny"])
def test_mxfp8_is_that_of_the_chain(ctas, kind, act):
    """Every code and scale, on data whose sums keep their size and on data whose sums cancel (in a flat image every output is
    open), by the whole grid and by one CTA."""
    shape = (1, 67, 133, 96) if ctas == 1 else (2, 200, 201, 128)
    for seed in range(1 if ctas == 1 else 4):
        x, w, b = data(kind, shape, 10 + seed)
        want = quantise(chain(x, w, b).view(-1, shape[3]), act)
        got, again = dw_mxfp8(x, w, b, act), dw_mxfp8(x, w, b, act)
        codes, scales = int((got[0] != want[0]).sum()), int((got[1] != want[1]).sum())
        assert codes == 0 and scales == 0, f"{codes} of {want[0].numel()} codes, {scales} of {want[1].numel()} scales differ"
        assert torch.equal(again[0], got[0]) and torch.equal(again[1], got[1])


def test_stack_on_chain_sums(ops, monkeypatch):
    """The refiner stack on four image pairs: the same bytes as with every depthwise layer summed by the chain."""
    import flashim_b200
    from flashim_b200 import refiner
    from flashim_b200.quant import swizzle_scales

    levels = ((50, 512), (100, 256), (200, 128))
    model = flashim_b200.load("refiner-stack", "fp8", device=DEV, engine="eager", overrides={"arch.levels": [list(v) for v in levels]})
    g = torch.Generator(device=DEV).manual_seed(9)
    pyramid = [torch.randn(8, size, size, c, generator=g, device=DEV).to(BF16) for size, c in levels]
    got = model(pyramid)

    class ChainSummed:
        def __getattr__(self, name):
            return getattr(ops, name)

        def depthwise5x5_act_mxfp8(self, value, weight, bias, act):
            pixels = value.permute(0, 2, 3, 1).contiguous()
            codes, scales = quantise(chain(pixels, weight, bias).view(-1, pixels.shape[3]), act)
            return codes.view(torch.float8_e4m3fn), swizzle_scales((scales.int() - 127).to(torch.int8))

    monkeypatch.setattr(refiner, "ops", ChainSummed())
    for mine, want in zip(got, model(pyramid)):
        assert same_bytes(mine, want)


def test_bits_do_not_depend_on_how_the_work_is_cut(ops):
    """Which steps are summed again as a whole is a matter of their own data, not of what a list holds already: areas that cancel
    in a few, in some and in most pixels of a step, on grids that cut the steps into different ranges and one image at a time."""
    from flashim_b200 import _native

    lib, shape = _native.library(), (4, 200, 201, 96)
    g = torch.Generator(device=DEV).manual_seed(6)
    density = torch.rand(shape[0], 1, 1, generator=g, device=DEV) * 0.002
    x, w, b = cancelling(shape, 7, torch.rand(shape[:3], generator=g, device=DEV) < density)
    image = x.permute(0, 3, 1, 2)
    want = ops.depthwise5x5_act(image, w, b, "none")
    try:
        for ctas in (1, 5, 40):
            lib.fim_dw_tune(ctas, 0)
            assert same_bytes(ops.depthwise5x5_act(image, w, b, "none"), want)
    finally:
        lib.fim_dw_tune(0, 0)
    for i in range(shape[0]):
        assert same_bytes(ops.depthwise5x5_act(x[i: i + 1].permute(0, 3, 1, 2), w, b, "none"), want[i: i + 1])
