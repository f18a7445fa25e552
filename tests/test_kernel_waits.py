"""Bounded waits of the kernels, read from their source.

Every lane that waits decides a time-out for itself (its own clock, its own look at the abort flag).  A role that one lane
plays may act on that; a warp whose lanes go on together to ``.sync`` instructions or warp barriers has to agree first, or
the lanes that stayed would wait for those that left.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sensenova_u1_b200" / "csrc"
FILES = sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"\b(mbar_wait|count_wait)", p.read_text()))
WAIT = re.compile(r"\b(mbar_wait|mbar_wait_cl|count_wait)\s*\(")
VOTE = "__all_sync(0xffffffffu, ok)"
ONE_LANE = re.compile(r"if\s*\([^{};]*\b(lane|threadIdx\.x) == 0[^{};]*\)\s*$")


def _unvoted(src: str):
    """Waits that are neither in a one-lane branch (or function) nor voted on, at once or before ``ok`` decides anything."""
    src = re.sub(r"//[^\n]*", "", src)
    found, stack, start = [], [], 0        # stack: is the enclosing block played by one lane
    for i, c in enumerate(src):
        if c == "{":
            stack.append(bool(ONE_LANE.search(src[start:i])) or (bool(stack) and stack[-1]))
            start = i + 1
        elif c == "}":
            stack.pop()
            start = i + 1
        elif c == ";":
            if re.match(r"\s*if \(threadIdx\.x != 0\) return$", src[start:i]) and stack:
                stack[-1] = True
            start = i + 1
        elif c in "mc" and stack and not stack[-1] and WAIT.match(src, i) and not re.match(r"\w", src[i - 1]):
            head = src[start:i]
            if re.search(r"__all_sync\(0xffffffffu,\s*$", head) or re.search(r"if \(lane == 0\) [\w ]+= $", head):
                continue
            if re.search(r"^\s*(if \([^()]*\)\s*)?(ok &=|bool ok =) $", head):
                used = re.search(r"\b(break|return)\b|\(!?ok\b|(&&|\|\|) !?ok\b", src[i:])
                if VOTE in src[i:i + used.end() if used else len(src)]:
                    continue
            found.append(src[i:src.index(")", i) + 1])
    return found


def test_the_reader_tells_the_forms_apart():
    assert len(_unvoted("void f() { if (lane == 0) { if (!mbar_wait(&a[0], 1)) return; } }")) == 0
    assert len(_unvoted("void f() { if (threadIdx.x != 0) return; while (x) { mbar_wait(a); } }")) == 0
    assert len(_unvoted("void f() { bool ok = __all_sync(0xffffffffu, mbar_wait(a, 0)); }")) == 0
    assert len(_unvoted("void f() { while (ok) { ok &= mbar_wait(a, 0); g(); ok = __all_sync(0xffffffffu, ok); } }")) == 0
    assert len(_unvoted("void f() { while (ok) { ok &= mbar_wait(a, 0); if (!ok) break; ok = __all_sync(0xffffffffu, ok); } }")) == 1
    assert len(_unvoted("void f() { ok &= mbar_wait(a, 0); if (x && ok) g(); }")) == 1
    assert len(_unvoted("void f() { if (lane == 0) { g(); } bool ok = mbar_wait(a, 0); }")) == 1
    assert len(_unvoted("void f() { if (rank == 0) { if (!count_wait(a, 0)) { break; } } }")) == 1


@pytest.mark.parametrize("name", FILES)
def test_whole_warps_vote_on_their_waits(name):
    src = (CSRC / name).read_text()
    src = re.sub(r"__device__ __forceinline__ bool (mbar_wait_cl|count_wait)\(.*?\n}\n", "", src, flags=re.S)   # definitions
    assert _unvoted(src) == []
