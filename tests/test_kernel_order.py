"""The order of writes that the evolve kernel's words rest on, read from its source: a row is
published by one thread of the group that wrote it, so that thread must first have met the
others.  No run shows a missing barrier reliably (the window is a warp held up for thousands
of cycles), and none is provoked."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-brkga_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def body(text, head):
    """the braces' contents that follow `head`"""
    at = text.index("{", text.index(head))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError(head)


def test_rows_end_with_the_group_together():
    row = body(source("row_body.cuh"), "void row_work(")
    assert row.rstrip().endswith("g.sync();")
    # a return after a store to the row: the stores start with the elite copy
    stores = row[row.index("build == BUILD_COPY"):]
    returns = [m.start() for m in re.finditer(r"\breturn;", stores)]
    assert returns
    for at in returns:
        assert stores[:at].rstrip().endswith("g.sync();")


def test_words_follow_row_work():
    """every release of a fitness word comes from the thread group's first thread, after row_work"""
    kernel = body(source("evolve.cu"), "evolve_kernel(EvolveArgs A)")
    releases = [m.start() for m in re.finditer(r"st\.release", kernel)]
    assert len(releases) == 2
    for at in releases:
        loop = kernel[kernel.rindex("for (int q = g.rg", 0, at):at]
        assert "row_work<" in loop and "if (g.tid == 0)" in loop[loop.index("row_work<"):]


def test_selection_stops_at_a_wait_that_ran_out():
    """a peel that gave up leaves a half-written front table: the kernels that place survivors by
    it start with the check"""
    text = source("nsga2.cu")
    assert "if (d.stuck) return false;" in body(text, "bool select_active(")
    kernels = ["nsga_peel_rows_kernel(PopDesc", "nsga_front_crowd_kernel(PopDesc", "nsga_cut_kernel(PopDesc",
               "nsga_order_kernel(PopDesc", "nsga_select_kernel(PopDesc"]
    for k in kernels:
        start = body(text, k)
        assert "select_active(" in start[:start.index("return;")], k
    kernel = body(source("evolve.cu"), "evolve_kernel(EvolveArgs A)")
    assert kernel.index("if (sd.stuck) return;") < kernel.index("stage_points")
