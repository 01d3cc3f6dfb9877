"""Launches that overlap: the order of the calls in the kernels' sources that no run on a GPU may put to the test (a kernel that
lets the next one start before it holds its tensor memory can wait for that one, which waits for it)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "flashim_b200" / "csrc"


def _kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        starts = [m.start() for m in re.finditer(r"__global__ void", text)]
        for begin, end in zip(starts, [*starts[1:], len(text)]):
            body = text[begin:end]
            yield pytest.param(body, id=f"{path.stem}-{re.search(r'(\w+_kernel)', body).group(1)}")


def _block(body: str, at: int) -> str:
    """The innermost braces around position ``at``, from there on."""
    depth = 0
    for i in range(at, len(body)):
        depth += {"{": 1, "}": -1}.get(body[i], 0)
        if depth < 0:
            return body[at:i]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("body", list(_kernels()))
def test_release_comes_behind_the_tensor_memory(body):
    releases, waits = [m.start() for m in re.finditer(r"grid_release\(\)", body)], [m.start() for m in re.finditer(r"grid_wait\(\)", body)]
    assert len(releases) == 1 and len(waits) == 1 and releases[0] < waits[0]
    allocations = [m.start() for m in re.finditer(r"tmem_alloc(?:_pair)?\(", body)]
    if not allocations:
        return
    assert max(allocations) < releases[0]
    branch = body.rindex("if (warp == 1) {", 0, min(allocations)) + len("if (warp == 1) {")
    assert "grid_release()" in _block(body, branch)  # by the warp that allocates
