"""Kernels that overlap the kernel before them (griddepcontrol.wait) read what
it writes: none may take a pointer that promises its memory does not change
while the kernel runs."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "g-mm-repair_gb300" / "csrc"


def _kernels():
    """(name, parameters, body) of every __global__ function."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^\n]*?\)\s+)?(\w+)\s*\(", text):
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params, at = text[m.end():at - 1], text.index("{", at)
            start, depth = at, 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
                if not depth:
                    break
            yield m.group(1), params, text[start:at]


def test_waiting_kernels_promise_nothing():
    waiting = {name: params for name, params, body in _kernels() if "wait_for_previous_kernel()" in body}
    assert {"k_level", "k_restride", "k_word_fold", "k_word_sum", "k_left_fold", "k_left_columns"} <= set(waiting)
    assert not [name for name, params in waiting.items() if "__restrict__" in params]
