"""Programmatic dependent launch (a kernel's blocks start while the one before it still
runs) is only sound when a kernel waits for the previous one before it touches memory
that kernel may write.  Read from the sources, since a missing wait is not run: where
yee_split.cu's kernels wait."""
from __future__ import annotations

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "3d_fdtd_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def body(text, start):
    """The braces' content that opens at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for e in range(i, len(text)):
        depth += (text[e] == "{") - (text[e] == "}")
        if depth == 0:
            return text[i + 1:e]
    raise AssertionError("unbalanced braces")


def test_split_step_kernels_wait_first():
    text = source("yee_split.cu")
    # the wait, then the trigger, on every path
    wait = body(text, text.index("void after_previous()"))
    assert re.sub(r"\s+", " ", wait).strip() == ('asm volatile("griddepcontrol.wait;" ::: "memory"); '
                                                 'asm volatile("griddepcontrol.launch_dependents;" ::: "memory");')
    assert text.count("griddepcontrol") == 2
    launched = set(re.findall(r"launch_cells\((\w+)<", text))
    assert launched == {"k_update_E", "k_update_H", "k_mur_step"}
    for k in launched:
        b = body(text, re.search(rf"\n{k}\(|void __launch_bounds__\(\w+\) {k}\(", text).end())
        first = [s.strip() for s in b.split(";")]
        first = [s for s in first if s and not s.startswith("using ")]
        assert first[0] == "after_previous()", (k, first[0])
