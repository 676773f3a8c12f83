"""What has to hold in the kernels' source and cannot be provoked on a GPU without a wait that hangs (CPU)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dhellam_b200" / "csrc"


def _uses_with_blocks(text, name):
    """``(line, headers of the enclosing blocks)`` of every call of ``name``."""
    text = re.sub(r"//[^\n]*", "", text)
    stack, start, calls = [], 0, {m.start() for m in re.finditer(rf"\b{name}(?:<[^<>()]*>)?\(", text)}
    for i, c in enumerate(text):
        if i in calls:
            yield text.count("\n", 0, i) + 1, [*stack, text[start:i]]
        if c == "{":
            stack.append(text[start:i])
        elif c == "}" and stack:
            stack.pop()
        if c in "{};":
            start = i + 1


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_a_wait_outside_a_single_lane_branch_has_one_answer_for_the_warp(path):
    """``mbar_wait`` answers lane by lane.  Where a whole warp waits, lanes must not part over a wait that gives up: votes and TMEM
    accesses behind it need all 32, so such a wait goes through ``warp_wait``."""
    lone = [line for line, blocks in _uses_with_blocks(path.read_text(), "mbar_wait")
            if not any(re.search(r"if \(.*(lane == 0|threadIdx\.x == 0)", b, re.S) for b in blocks)]
    assert not lone, f"{path.name}: per-lane waits of a whole warp in lines {lone}"


def test_the_small_gemm_leaves_the_output_alone_when_a_wait_ran_out():
    """All stores of ``gemm_small_kernel`` to the output stand where no CTA of the cluster has given up: without its partial tile the
    sums would be of whatever the shared memory held."""
    text = (CSRC / "gemm_sm100.cu").read_text()
    body = text[text.index("\ngemm_small_kernel("):text.index("static int launch_small(")]
    uses = [blocks for _, blocks in _uses_with_blocks(body.replace("p.d)", "output_of(p))"), "output_of")]
    assert len(uses) == 2 and all(any("gave_up == 0" in b for b in blocks) for blocks in uses)
