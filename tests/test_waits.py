"""The bounded waits of the kernels, by reading their source: a warp gives up
as one, never a lane by itself beside lanes that go on to a warp-wide vote."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "libmarshal_gb300", "csrc")


def _loops(text):
    """Bodies of the while loops (with braces) of a source text."""
    for m in re.finditer(r"\bwhile\s*\(", text):
        i, depth = m.end(), 1
        while depth:  # the condition
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        j = i + len(text[i:]) - len(text[i:].lstrip())
        if j >= len(text) or text[j] != "{":
            continue
        k, depth = j + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield text.count("\n", 0, m.start()) + 1, text[j:k]


@pytest.mark.parametrize("path", sorted(
    os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu"))))
def test_loops_with_votes_end_for_the_whole_warp(path):
    text = open(os.path.join(CSRC, path)).read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/",
                  lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)
    for line, body in _loops(text):
        if not re.search(r"__(ballot|any|all|shfl)_sync|__shfl_\w+_sync", body):
            continue
        for test in re.finditer(r"if \(([^;{]*)\)\s*(\{[^{}]*\bbreak;|break;)",
                                body):
            if "global_timer_ns" in test.group(1):
                assert re.search(r"__(any|all|ballot)_sync", test.group(1)), \
                    "%s:%d: a lane leaves by its own clock" % (path, line)
