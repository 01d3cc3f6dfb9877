"""Generates ``gelu_table.inc``: GELU (erf form) of every bf16 value as a table the conv epilogue looks up.

The conv epilogue applies GELU to a value that has just been rounded to bf16 and rounds the result to bf16 again, so
GELU there is a function from 65536 bit patterns to 65536 bit patterns. torch's own result
(``F.gelu(x.float()).to(torch.bfloat16)``, the expression FlashIM's reference epilogues use, flashim/ops/gemm.py:93-95)
is tabulated over the magnitudes where it is neither ``x / 2`` (tiny ``|x|``), ``x`` (large positive) nor ``-0`` (large
negative); the kernel reproduces it exactly, without evaluating erf.

Table entry ``t`` (one 32-bit word): low half = delta for ``x >= 0``, high half = delta for ``x < 0``, where the
magnitude bits of the result are ``max(a + delta, 0)`` for input magnitude bits ``a`` (16-bit signed arithmetic) and the
sign bit of the result is the sign bit of the input. ``t = clamp(a - (BASE - 1), 0, ENTRIES - 1)``: entry 0 serves every
magnitude below BASE (delta -0x80: the exponent drops by one, magnitudes below the smallest normal number become zero)
and the last entry every magnitude from TOP on (delta 0 for positive values, -0x8000 for negative ones: zero).

The epilogues that requantise to E4M3 evaluate GELU by arithmetic instead (``gelu_arithmetic_bf16x2`` in conv.cu). ``verify_arithmetic``
restates it with the coefficients read from that source: for every bf16 value from ``EXACT_FROM`` up the result is torch's, and below
the E4M3 codes of the two are the same under every exponent from ``CODES_FROM`` up but for the values in ``EXCEPTIONS``, whose upper
neighbours have the right codes there and under every exponent not more than ``REPLACED_BELOW`` less, with room for the error of the
evaluation. The coefficients are a point of the polytope these conditions span (each bounds log2 of Phi(-|x|),
which is linear in them, from both sides), found by linear programming with the largest distance from all of its sides.

Run ``python flashim_b200/csrc/make_gelu_table.py`` to rewrite the file; ``--check`` only verifies the committed one.
Deviations from torch that the check allows: subnormal bf16 inputs (flushed to zero), NaN payloads, and the top binade
(``|x| >= 2**127``), where torch's own expression overflows to infinity.
"""

from __future__ import annotations

import re
import sys
from pathlib import Path

import torch
import torch.nn.functional as F

OUT = Path(__file__).resolve().parent / "gelu_table.inc"


def torch_gelu_bits() -> tuple[torch.Tensor, torch.Tensor]:
    bits = torch.arange(65536, dtype=torch.int32)
    x = bits.to(torch.int16).view(torch.bfloat16)
    y = F.gelu(x.float()).to(torch.bfloat16)
    return bits, y.view(torch.int16).to(torch.int32) & 0xFFFF


def build() -> tuple[int, int, list[int]]:
    bits, out = torch_gelu_bits()
    a, mag, negative = bits & 0x7FFF, out & 0x7FFF, bits >= 0x8000
    normal = (a >= 0x100) & (a < 0x7F00)
    simple = torch.where(a < 0x4000, mag == (a - 0x80).clamp(min=0), torch.where(negative, mag == 0, mag == a))
    hard = a[normal & ~simple]
    base, top = int(hard.min()), int(hard.max()) + 1
    # every magnitude in [base, top) gets an entry; both signs share the index
    words = [(0x10000 - 0x80) | ((0x10000 - 0x80) << 16)]
    for value in range(base, top):
        dp = (int(mag[value]) - value) & 0xFFFF
        dn = (int(mag[value | 0x8000]) - value) & 0xFFFF
        words.append(dp | (dn << 16))
    words.append(0x0000 | (0x8000 << 16))
    return base, top, words


def emulate(base: int, words: list[int]) -> torch.Tensor:
    """The kernel's integer arithmetic on all 65536 inputs."""
    bits = torch.arange(65536, dtype=torch.int64)
    a = bits & 0x7FFF
    t = (a - (base - 1)).clamp(0, len(words) - 1)
    table = torch.tensor(words, dtype=torch.int64)
    word = table[t]
    delta = torch.where(bits >= 0x8000, word >> 16, word & 0xFFFF)
    delta = torch.where(delta >= 0x8000, delta - 0x10000, delta)
    return (a + delta).clamp(min=0) | (bits & 0x8000)


def verify(base: int, words: list[int]) -> None:
    bits, want = torch_gelu_bits()
    got = emulate(base, words).to(torch.int32)
    a = bits & 0x7FFF
    checked = (a >= 0x100) & (a < 0x7F00)
    assert torch.equal(got[checked], want[checked]), "table does not reproduce torch's GELU"
    assert int(got[0]) == 0 and int(got[0x8000]) == 0x8000  # zeros keep their sign
    assert int(got[0x7F80]) == 0x7F80  # +inf


EXACT_FROM, CODES_FROM, EXCEPTIONS, REPLACED_BELOW = -3.515625, -9, {-6: -4.5, -2: -3.53125}, 2
P_ERROR = 1.5e-6  # relative: the last roundings of q (|q| <= 13, and half an ulp of it in the exponent) and of ex2.approx (2**-22)


def verify_arithmetic() -> None:
    text = (OUT.parent / "conv.cu").read_text()
    body = text[text.index("gelu_arithmetic_bf16x2(uint32_t r) {"):]
    numbers = re.findall(r"pack2\((-?\d\.\d+e[-+]\d+)f, \1f\)", body[: body.index("ex2_approx")])
    coefficients = [torch.tensor(float(n), dtype=torch.float32) for n in numbers]
    assert len(coefficients) == 6
    exceptions = re.search(r"gelu_exception\(int e\) { return e == (-\d+) \? (0x\w+)u : (0x\w+)u; }", text)
    as_float = lambda code: float(torch.tensor([int(code, 16) - 0x10000], dtype=torch.int16).view(torch.bfloat16))  # noqa: E731
    assert {int(exceptions[1]): as_float(exceptions[2]), -2: as_float(exceptions[3])} == EXCEPTIONS
    bits, want = torch_gelu_bits()
    x = bits.to(torch.int16).view(torch.bfloat16).float()
    u, relu = torch.minimum(x, -x), torch.where(bits >= 0x8000, torch.tensor(-0.0), x)
    q = coefficients[0].expand(65536)
    for c in coefficients[1:]:
        q = (q.double() * u.double() + c.double()).float()  # one rounding, as an fma
    a = bits & 0x7FFF
    checked = (a >= 0x100) & (a < 0x7F00)
    expected = want.to(torch.int16).view(torch.bfloat16)
    for error in (-P_ERROR, 0.0, P_ERROR):
        p = torch.where(q < -126, torch.tensor(0.0, dtype=torch.float64), torch.exp2(q.double()) * (1 + error))
        value = (u.double() * p + relu.double()).float()
        value = torch.where((p == 0) & (bits >= 0x8000), torch.tensor(-0.0), value)
        got = value.to(torch.bfloat16)
        same = (got.view(torch.int16).to(torch.int32) & 0xFFFF) == want
        assert bool(same[checked & (x >= EXACT_FROM)].all()), "not exact"
        for e in range(CODES_FROM, 128):
            codes = [(t.double() * 2.0 ** -e).clamp(-448, 448).float().to(torch.float8_e4m3fn).view(torch.uint8) for t in (got, expected)]
            differ = checked & (codes[0] != codes[1])
            assert not bool((differ & (x != EXCEPTIONS.get(e, 1e30))).any()), f"codes differ under the exponent {e}"
            for exponent, value in EXCEPTIONS.items():
                at = int((x == value).nonzero())
                assert e < exponent - REPLACED_BELOW or codes[0][at - 1] == codes[1][at], f"the neighbour of {value} under the exponent {e}"


def render(base: int, top: int, words: list[int]) -> str:
    lines = [
        "// Generated by make_gelu_table.py from torch's erf-form GELU; do not edit.",
        f"constexpr int kGeluBase = 0x{base:04X};     // first bf16 magnitude with a table entry of its own",
        f"constexpr int kGeluEntries = {len(words)};  // entry 0: magnitudes below kGeluBase; last entry: 0x{top:04X} and above",
        "__device__ const uint32_t kGeluTable[kGeluEntries] = {",
    ]
    for i in range(0, len(words), 8):
        lines.append("    " + ", ".join(f"0x{w:08X}u" for w in words[i: i + 8]) + ",")
    lines.append("};")
    return "\n".join(lines) + "\n"


def main() -> None:
    base, top, words = build()
    verify(base, words)
    verify_arithmetic()
    text = render(base, top, words)
    if "--check" in sys.argv:
        assert OUT.read_text() == text, f"{OUT.name} is stale: run make_gelu_table.py"
        print(f"{OUT.name} ok: base 0x{base:04X}, {len(words)} entries")
        return
    OUT.write_text(text)
    print(f"wrote {OUT} (base 0x{base:04X}, top 0x{top:04X}, {len(words)} entries, {4 * len(words)} bytes)")


if __name__ == "__main__":
    main()
