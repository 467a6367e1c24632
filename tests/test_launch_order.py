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


def test_read_only_loads_take_only_what_no_step_writes():
    # the read-only path (__ldg) is for data that nothing writes while the kernel lives, and a
    # kernel started programmatically lives while the launch before it still writes fields,
    # auxiliaries and source planes: coefficients and profiles only
    constant = re.compile(r"a\.(prof\[[^\]]+\]\[[^\]]+\]|c[ab]\[[^\]]+\]) \+ ")
    seen = 0
    for name in ("yee_tile.cu", "tile_cells.cuh", "yee_stream.cu", "stream_cells.cuh", "yee_flat4.cu", "flat4_cells.cuh",
                 "yee_flat.cu", "yee_split.cu", "yee_wave.cu", "yee_sweep.cu", "aux_kernels.cu", "plane_ops.cuh"):
        text = source(name)
        if name == "flat4_cells.cuh":   # the vector form of the load itself
            start = text.index("Vf<W> ldv(")
            text = text.replace(body(text, start), "", 1)
            text = text.replace("Vf<W> ldv(", "", 1)
        for arg in re.findall(r"(?:__ldg|\bldv<\w+>)\(([^;]*?)\)[,;\s]", text):
            assert constant.match(arg), (name, arg)
            seen += 1
        assert "ld.global.nc" not in text
    assert seen > 10


def test_tables_read_before_the_wait_are_uploaded_and_waited_for():
    # a tile's block reads its box and the CPML profiles before it waits for the previous
    # launch: the host waits for their copies before it enqueues any
    text = source("engine.cu")
    for f in ("bool build_profiles(Grid *g, double dt)", "bool tile_prepare(Grid *g)"):
        b = body(text, text.index(f))
        assert "cudaStreamSynchronize(g->st)" in b[b.rindex("cudaMemcpyAsync"):], f
