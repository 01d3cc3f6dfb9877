"""The GELU by arithmetic of the epilogues that requantise to E4M3 against the table of torch's results (flag 1024: the general
epilogue), over every bf16 argument. The arguments are biases under products of zeros."""

import pytest
import torch

from fim_testlib import DEV, conv_schedule, same_bytes, to_dev

pytestmark = pytest.mark.gpu
E4M3, BF16 = torch.float8_e4m3fn, torch.bfloat16
POINT = (1, 1, 1, 1, 0, 0, 1, 1)
TAIL = torch.cat((torch.arange(0xC05C, 0xC0C0), torch.tensor([0xC0FF, 0xC13F, 0xC2C8, 0xFF7F]))).to(torch.int32)  # -3.4 to -6, and far out


@pytest.fixture(scope="module")
def fused():
    import flashim_b200

    yield flashim_b200.ops.mxfp8_conv2d_fused
    flashim_b200.ops.reset_call_counts()  # other modules count calls


def values(bits):
    return bits.to(torch.int16).view(BF16)


def normal(bias):
    """Results of arguments below 2**-125 are subnormal: the table gives zero or half the bits, the arithmetic torch's rounding."""
    magnitude = bias.view(torch.int16).to(torch.int32) & 0x7FFF
    return (magnitude == 0) | (magnitude >= 0x100)


def both(fused, bias, geometry=POINT, shape=(1, 1, 5), cin=128, **kw):
    k = geometry[0] * geometry[1] * cin
    args = to_dev(torch.zeros(*shape, cin).to(E4M3), torch.zeros(cin // 32, dtype=torch.int8), torch.zeros(bias.numel(), k).to(E4M3),
                  torch.zeros((bias.numel() + 127) // 128 * 128 * ((k // 32 + 3) // 4) * 4, dtype=torch.uint8), bias)
    outs = []
    for flags in (0, 1024):
        with conv_schedule(0, 0, flags):
            out = fused(*args, *geometry, act="gelu", **kw)
            outs.append(out if isinstance(out, tuple) else (out,))
    return outs


@pytest.mark.parametrize("order", ["by bits", "shuffled"])
def test_every_argument_under_static_exponents(fused, order):
    bits = torch.arange(65536, dtype=torch.int32)
    if order == "shuffled":
        bits = bits[torch.randperm(65536, generator=torch.Generator().manual_seed(1))]
    for e in (-127, -20, *range(-12, 3), 60):
        for part in bits.view(8, 8192):
            bias = values(part)
            got, want = both(fused, bias, out_exponent=torch.full((256,), e, dtype=torch.int8, device=DEV))
            keep = normal(bias).to(DEV)
            assert same_bytes(got[0][..., keep], want[0][..., keep]), e


def test_halo_patches(fused):
    exponents = torch.tensor([-6, -2], dtype=torch.int8, device=DEV)
    for part in TAIL[: 96].view(3, 32):
        got, want = both(fused, values(part.repeat(2)), (3, 3, 1, 1, 1, 1, 1, 1), (1, 17, 9), 64, out_exponent=exponents)
        assert same_bytes(got[0], want[0])


def test_blocks_with_exponents_of_their_own(fused):
    """One value that sets the exponent, from -40 to 4, beside arguments where torch's result is noise; values that are not finite."""
    g = torch.Generator().manual_seed(2)
    blocks = []
    for e in range(-40, 5):
        for mantissa in (1.01, 1.74, 1.76):
            rest = TAIL[torch.randint(0, TAIL.numel(), (31,), generator=g)]
            top = torch.tensor([mantissa * 2.0 ** (e + 8)]).to(BF16).view(torch.int16).to(torch.int32)
            blocks.append(torch.cat((rest, top))[torch.randperm(32, generator=g)])
    for special in (0x7F80, 0xFF80, 0x7FC0, 0xFFC0):
        block = torch.randint(0x3E00, 0x4000, (32,), generator=g, dtype=torch.int32)
        block[7] = special
        blocks.append(block)
    bits = torch.stack(blocks).flatten()
    bias = values(torch.cat((bits, torch.zeros(-bits.numel() % 256, dtype=torch.int32))))
    got, want = both(fused, bias, dynamic_out=True)
    assert same_bytes(got[1], want[1]) and same_bytes(got[0], want[0])
