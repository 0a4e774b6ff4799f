"""The attention core's warps wait lane by lane and go on together. A barrier poll is each lane's own, so
lanes may part at a wait, as they do where rows past the end are left out; tcgen05.ld and tcgen05.st are
instructions of the whole warp and need them back. No run tells a warp that was brought together from one
that happened to be, so this reads the kernel's source: between a parting and what needs the whole warp
stands a join."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "foldjax_b200" / "csrc" / "triatt_core.cu"
WAIT = r"\bmbar_(?:wait|test)\("
JOIN = r"\b__syncwarp\(\)|\b__(?:all|any)_sync\("
TMEM = r"\btmem_(?:ld|st)\d+\("


def _roles():
    """The kernel's text of the warps that load and issue, and of those that do the softmax."""
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    text = text[text.index("setmaxnreg.dec"):text.index("mask_bias_kernel(")]
    return text.split("setmaxnreg.inc")


def _not_joined(text, needs):
    """Every ``needs`` that is reached from a wait or a ragged row's end without a join, in source order,
    with the parting."""
    found, parted = [], None
    for m in re.finditer(rf"(?P<part>{WAIT}|\bif \(in_range)|(?P<join>{JOIN})|{needs}", text):
        if m.lastgroup == "part":
            parted = text[m.start():text.index("\n", m.start())]
        elif m.lastgroup == "join":
            parted = None
        elif parted:
            found.append((parted, m.group()))
    return found


def test_tensor_memory_is_accessed_by_joined_warps():
    softmax = _roles()[1]
    assert len(re.findall(WAIT, softmax)) >= 6 and len(re.findall(TMEM, softmax)) >= 10
    assert not _not_joined(softmax, TMEM)


def test_issuing_lane_does_not_run_ahead_of_its_warp():
    """All lanes of the loading and issuing warps wait on barriers that tell two phases apart, and one lane
    makes the next phase come: it may pass a wait only together with the others. No lane leaves the loops
    before the others, which would wait for it at a join."""
    control = _roles()[0]
    issued = r"\bif \([^)]*\bleader\b"
    assert len(re.findall(issued, control)) == 6
    assert not _not_joined(control, issued)
    assert "break" not in control and "return" not in control
    assert not re.search(r"for \([^;]*;[^;]*alive", control)
