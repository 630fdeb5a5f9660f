"""Bounded waits of whole warps in the fused kernels (``csrc/fused``), read from their source: a wait that can run out is either
one thread's, or all lanes of the warp act on one answer. A lane that leaves a loop alone would never be met in the warp-wide
instructions of the others, and the bounded wait would have no end. (Making a wait run out in a kernel that is multiplying is
nothing to try on a device.)"""
import re
from pathlib import Path

import pytest

FUSED = Path(__file__).resolve().parent.parent / "csrc" / "fused"


def _calls(text):
    """(name, start of its statement, headers of the enclosing blocks) of every mbarrier wait."""
    text = re.sub(r"//[^\n]*", "", text)
    stack, last = [], 0
    for m in re.finditer(r"[{};]|\bmbar_wait(?:_warp)?\(", text):
        tok = m.group()
        if tok == "{":
            stack.append(text[last:m.start()].strip())
        elif tok == "}":
            stack.pop()
        elif tok != ";":
            yield tok[:-1], text[last:m.start()].strip(), list(stack)
            continue
        last = m.end()


@pytest.mark.parametrize("name", ["tp_gemm.cu", "tp_skinny.cu"])
def test_lanes_of_a_warp_act_on_one_answer(name):
    seen = {"one": 0, "warp": 0}
    for call, statement, headers in _calls((FUSED / name).read_text()):
        one_thread = any(re.search(r"elect_one\(\)|threadIdx\.x == 0", h) for h in headers)
        if call == "mbar_wait_warp":
            assert not one_thread, statement      # a vote that one thread holds alone never ends
            seen["warp"] += 1
        elif one_thread:
            seen["one"] += 1
        else:
            # no lane may leave on its own answer: it is dropped, and the flag of the wait that ran out is asked later, by all
            assert statement == "(void)", f"a warp's lanes each act on their own: {statement} {call}("
            seen["warp"] += 1
    assert seen["one"] >= 3 and seen["warp"] >= 3
