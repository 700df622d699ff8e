"""The waits of k_resident, read from their source on the CPU: a warp's lanes may see different values of a
word that another warp or another block writes, and the code behind a wait holds full-mask collectives, so
every such read that decides whether a wait ends goes through a vote of the whole warp."""
import os
import re

import pytest

from conftest import ROOT

SOURCE = open(os.path.join(ROOT, "h2_b200", "csrc", "h2g_resident.cuh")).read()


def closing(text, start, pair):
    """Index behind the bracket that closes the one at `start`."""
    depth = 0
    for q in range(start, len(text)):
        depth += (text[q] == pair[0]) - (text[q] == pair[1])
        if depth == 0:
            return q + 1
    raise AssertionError("unbalanced")


def body(name):
    m = re.search(r"__device__ __forceinline__ \w+ " + name + r"\(", SOURCE)
    assert m, name
    start = SOURCE.index("{", closing(SOURCE, m.end() - 1, "()"))
    return re.sub(r"//[^\n]*", "", SOURCE[start:closing(SOURCE, start, "{}")])


def without_votes(text):
    while True:
        m = re.search(r"__(any|all)_sync\(", text)
        if not m:
            return text
        text = text[:m.start()] + text[closing(text, m.end() - 1, "()"):]


@pytest.mark.parametrize("name,reads", [("rs_planes_ready", ["rs_progress"]), ("rs_wait_planes", ["rs_progress"]),
                                        ("rs_wait", ["rows_missing", "edges_missing"]),
                                        ("rs_wait_edges", ["edges_missing"]), ("rs_give_up", ["ld_relaxed_s32"])])
def test_a_wait_ends_for_the_whole_warp(name, reads):
    text = without_votes(body(name))
    for word in reads:
        assert word + "(" not in text, (name, word)


def test_no_read_only_load_of_a_vector_that_the_launch_writes():
    """Read-only loads (ld.global.nc) may return old values of memory that the same launch writes.  k_resident
    writes v in stages 1 and 2, q (as y) in stage 1, xx and the row sums; the SOR kernel writes xx."""
    code = re.sub(r"//[^\n]*", "", SOURCE)
    resident = code[code.index(" k_resident("):code.index(" k_resident_sor(") if " k_resident_sor(" in code else None]
    for vector in ("A.v", "A.y", "A.xx", "A.rowsum", "A.partials"):
        assert "__ldg(" + vector not in resident, vector
    for m in re.finditer(r"__ldg\(A\.q\b", resident):
        assert resident[:m.start()].rstrip().endswith("VM == 1 ? ld_once(A.q + ci) :")
    sor = code[code.index("k_resident_sor("):]
    for vector in ("A.xx", "A.rowsum", "A.partials"):
        assert "__ldg(" + vector not in sor, vector
