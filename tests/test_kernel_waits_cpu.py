"""Bounded waits of the kernels, read in their source: where all lanes of a warp wait, no lane may leave a loop on its own answer.

A lane that gave up would be missing at the votes, shuffles and warp barriers of the others, which wait for it without a limit; no run
on a GPU may show that, so the source is checked."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tunix_b200" / "csrc"
# blocks that one thread runs: their conditions, and functions that such a block calls
ONE_THREAD = re.compile(r"elect_one\(\)|\btid == \d+\b|\bthreadIdx\.x == 0\b|\blane == 0\b")
CALLED_BY_ONE = re.compile(r"\bissue_upto = |\bcopier_role\(|^\s*#define ")
LEAVES = re.compile(r"\b(break|return|continue)\b|\bok = false\b")


def _strip(text):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)
    return re.sub(r"^#(define (?:.*\\\n)*.*|undef .*|include .*|pragma .*)", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.M)


def lane_wise_exits(text):
    """Lines with a lane-wise wait whose failure leaves a loop or function, outside of the blocks of single threads. A macro whose
    name ends in _WAIT is such a wait."""
    text, found = _strip(text), []
    headers, last = [], 0                       # text in front of every open brace
    for m in re.finditer(r"[{};]|\bmbar_wait_bounded\(|\b[A-Z]+_WAIT\(", text):
        if m.group() == "{":
            headers.append(text[last:m.start()])
            last = m.end()
        elif m.group() == "}":
            headers and headers.pop()
            last = m.end()
        elif m.group() == ";":
            last = m.end()
        elif not any(ONE_THREAD.search(h) or CALLED_BY_ONE.search(h) for h in headers):
            head = text[last:m.start()]
            after = text[m.start():].split(";", 1)[0]           # up to the end of the statement, or into the block of an `if`
            macro = not m.group().startswith("mbar")
            if "__all_sync" in head or "bool mbar_wait" in head:
                continue
            if macro or (re.search(r"\bif \([^{;]*$", head) and LEAVES.search(after)):
                found.append(text.count("\n", 0, m.start()) + 1)
    return found


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_lanes_leave_waits_together(name):
    assert lane_wise_exits((CSRC / name).read_text()) == []


def test_the_reader_sees_lane_wise_exits():
    loop = "for (int i = 0; i < n; ++i) {{ {} tmem_ld(x); }}"
    for bad in ("if (!mbar_wait_bounded(b, i & 1, f, s, 1)) { ok = false; break; }", "if (!mbar_wait_bounded(b, 0, f, s, 1)) return;",
                "if (more &&\n !mbar_wait_bounded(b, 0, f, s, 1)) break;", "ROW_WAIT(b, i & 1, 1);"):
        assert lane_wise_exits(loop.format(bad)) and lane_wise_exits("} else { " + loop.format(bad) + " }")
        assert not lane_wise_exits("if (nit > 0 && elect_one()) { " + loop.format(bad) + " }")
    for good in ("if (!mbar_wait_warp(b, 0, f, s, 1)) break;", "ok = __all_sync(0xffffffffu, mbar_wait_bounded(b, 0, f, s, 1)); if (!ok) break;",
                 "const bool here = mbar_wait_bounded(b, 0, f, s, 1);"):
        assert not lane_wise_exits(loop.format(good))
