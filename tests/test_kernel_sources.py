"""Properties of kernels that are read off their source: what no test can
bring about on a device."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "flowpsi_b200" / "csrc"


def _body(text: str, start: str) -> str:
    """from start through the brace that closes the first one after it"""
    i = text.index(start)
    depth = 0
    for j in range(text.index("{", i), len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise ValueError(start)


def test_the_line_solve_gives_up_as_a_warp():
    """The walking warp's lanes wait one by one, and a bounded wait may give up
    in one lane alone.  The loops behind it hold warp-wide votes and barriers,
    so the warp has to go on or stop as one: the outcome is a vote."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "lsgs.cu").read_text())
    kernel = _body(text, "k_lsgs_thomas(int nst")
    copying = _body(kernel, "if (warp == 1)")
    walking = kernel[kernel.index(copying) + len(copying):]
    assert re.search(r"__all_sync\(0xffffffffu, wait\(", walking)
    bare = re.findall(r"(?<!__all_sync\(0xffffffffu, )(?<![\w_])wait\(", walking)
    assert not bare, f"{len(bare)} waits of the walking warp without a vote"
    # what the loops run on is set from those outcomes only
    for m in re.finditer(r"\bok\s*=\s*([^;]+);", walking):
        assert m.group(1) == "true" or m.group(1).startswith("wait_all("), m.group(0)
