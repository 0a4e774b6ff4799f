"""The general attention cores' products and what they read and overwrite. In the bf16 core a row's scores go to tensor memory that the
probabilities of the step before still occupy. Products of different shapes into different accumulators have no
order among each other that the instruction set promises, so the warp that issues scores first waits for the products
that read those probabilities. No run tells an order that was waited for from one that the
hardware happens to keep, so this reads the kernels' source. In both cores whole warps wait and one lane issues (test_core_joined_waits.py).
"""

import re
from pathlib import Path

from test_core_joined_waits import _not_joined

SOURCE = Path(__file__).resolve().parents[1] / "foldjax_b200" / "csrc" / "att_split.cu"


def _control():
    """The bf16 kernel's text of the warps that load and issue, one piece for each role."""
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    text = text[text.index("att_bf16_kernel("):]
    text = text[text.index("setmaxnreg.dec"):text.index("setmaxnreg.inc")]
    return re.split(r"\belse if \(warp\b", text)


def _float32_issuers():
    """The same of the float32 kernel's warps that issue (its producer is a single lane)."""
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    text = text[text.index("att_split_kernel("):text.index("att_bf16_kernel(")]
    text = text[text.index("else if (warp == 1)"):text.index("else if (warp >= 4)")]
    return re.split(r"\belse if \(warp\b", text)[1:]


def test_scores_wait_for_the_products_that_read_the_probabilities():
    scores = [role for role in _control() if "umma_bf16_ss(" in role]
    values = [role for role in _control() if "umma_bf16_ts(" in role]
    assert len(scores) == 1 and len(values) == 1 and scores != values
    rows = scores[0][scores[0].rindex("for (int wg"):]
    wait = r"mbar_wait\(&sm\.pv_done\[wg\], \(g & 1\) \^ 1,"
    assert re.search(wait, rows[:rows.index("umma_bf16_ss(")])
    assert re.search(r"umma_bf16_ts\([^;]*;\s*umma_commit\(&sm\.pv_done\[wg\]\);", values[0])


def test_issuing_lane_does_not_run_ahead_of_its_warp():
    issuers = _float32_issuers()
    assert len(issuers) == 2 and all("umma_bf16_" in role and "mbar_wait(" in role for role in issuers)
    for role in _control() + issuers:
        assert not _not_joined(role, r"\bif \([^)]*\bleader\b")
        assert "break" not in role and "return" not in role
