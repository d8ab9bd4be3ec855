"""The cell counts are zero when a rebuild chain starts: k_wrap_bin counts the
atoms up and k_scatter down again.  An error return between the two would leave
the counts for the next chain, whose scatter would then write past the order
array; so nothing that can fail may stand there (the scan's scratch is allocated
with the cells).  Read from the source: the failing case cannot be run."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exastamp_gb300", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def _body(src, head):
    start = src.index("{", src.index(head))
    depth = 0
    for k in range(start, len(src)):
        depth += (src[k] == "{") - (src[k] == "}")
        if depth == 0:
            return src[start:k + 1]
    raise AssertionError("unbalanced braces after " + head)


def test_nothing_can_fail_between_the_count_and_the_scatter():
    src = _code("gbmd_neighbors.cu")
    chain = _body(src, "static int rebuild_chain(")
    up, down = chain.index("k_wrap_bin<<<"), chain.index("k_scatter<<<")
    assert up < down
    between = chain[up:down]
    assert not re.search(r"\breturn\b|GBMD_CUDA|alloc\(", between)
    assert "scan(" in between
    scan = re.search(r"static (\w+) scan\(", src)
    assert scan.group(1) == "void" and "alloc(" not in _body(src, scan.group(0))


def test_a_failed_allocation_leaves_no_capacity():
    src = _code("gbmd_neighbors.cu")
    for head, cap in (("static int ensure_cells(", "cells_cap = 0"), ("static int build_list(", "nbr_cap = 0"),
                      ("static int filter_list(", "nbr_cap = 0")):
        body = _body(src, head)
        assert body.index(cap) < body.index("alloc(")
