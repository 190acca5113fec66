"""Rules of the programmatic launches that no run can show: a kernel placed
while its predecessor still runs must not hold what the predecessor waits for
(CPU; reads the kernel sources)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rapidfem_b200", "csrc")


def _source(name):
    """A source file without its comments."""
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def _body(src, start):
    """The brace-balanced block that opens at or after `start`."""
    i = src.index("{", start)
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j + 1]
    raise AssertionError("unbalanced braces")


def test_a_stage_holds_its_tmem_before_it_lets_the_next_launch_in():
    src = _source("rhs_tc.cuh")
    body = _body(src, src.index("rhs_tc_kernel(RhsParams"))
    alloc = body.index("tmem_alloc(")
    barrier = body.index("__syncthreads()", alloc)
    launch = body.index("pdl_launch()")
    assert alloc < barrier < launch < body.index("pdl_wait()")
    assert body.count("pdl_launch()") == 1
