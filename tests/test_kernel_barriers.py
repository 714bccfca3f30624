"""Barriers that a shared-memory table needs, checked in the kernels' source: a missing one is a race
that no run shows reliably."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "ckmpm_b200" / "csrc" / "kernels.cuh").read_text()


def without_constexpr_branches(text: str) -> str:
    """The text without the bodies of `if constexpr`: some instantiations do not have them."""
    out, at = "", 0
    for m in re.finditer(r"if constexpr \([^{;]*\) \{", text):
        if m.start() < at:
            continue
        out += text[at:m.start()]
        depth, at = 1, m.end()
        while at < len(text) and depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
    return out + text[at:]


CALLS = [m.start() for m in re.finditer(r"^  load_classes\(", SOURCE, re.M)]


@pytest.mark.parametrize("call", CALLS)
def test_colour_classes_are_read_after_a_barrier(call):
    """load_classes fills the colour classes from 8 threads; in every instantiation a barrier of the CTA
    comes before the first lookup by another lane."""
    use = re.compile(r"incoming_groups\(sc,|traversal_index\(sc,").search(SOURCE, call)
    assert use
    assert "__syncthreads();" in without_constexpr_branches(SOURCE[call:use.start()])


def test_every_kernel_with_colour_classes_is_checked():
    assert len(CALLS) == 4
