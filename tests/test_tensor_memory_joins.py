"""Tensor memory is accessed by whole warps, but a barrier poll is each lane's own: in every kernel a join stands
between a wait and the accesses behind it. No run tells a warp that was brought together from one that happened to
be, so this reads the kernels' sources. (The attention core has a test of its own, test_core_joined_waits.py; the
products' epilogues join in Accum::load, which every access of theirs goes through.)"""

import re
from pathlib import Path

import pytest

from test_core_joined_waits import TMEM, WAIT

CSRC = Path(__file__).resolve().parents[1] / "foldjax_b200" / "csrc"
FILES = ["att_split.cu", "pair_transition.cu", "single_attention.cu", "triatt_finish.cu", "triatt_project.cu", "trimul_contract.cu",
         "trimul_finish.cu", "trimul_project.cu"]
VOTED = r"(?:__all_sync\(0xffffffffu|named_barrier_and\([^,]*, 128), mbar_wait\("  # a wait and its join in one
JOIN = r"\b__syncwarp\(\)|\b__(?:all|any)_sync\(|\bnamed_barrier\(|\bif \(warp\b"  # (or another role's text begins)


@pytest.mark.parametrize("name", FILES)
def test_accesses_are_the_whole_warps(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    assert re.search(TMEM, text)
    found, parted = [], None
    for m in re.finditer(rf"(?P<join>{VOTED}|{JOIN})|(?P<part>{WAIT})|(?P<access>{TMEM}|\btake_pv\(\))", text):
        if m.lastgroup == "access" and parted:
            found.append((parted, m.group()))
        elif m.lastgroup != "access":
            parted = text[m.start():text.index("\n", m.start())] if m.lastgroup == "part" else None
    assert not found
