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


# Parameters of such kernels that only the host writes (before any of them starts).
HOST_WRITTEN = {"k_gather_f32": {"idx"}, "k_functionals": {"ptr", "idx", "w"}, "k_kcl_record_fun": {"ptr", "idx", "w"}}
FILES = ("dgtd_capi.cu", "kcl.cuh", "krylov.cuh", "rhs_fp32.cuh", "rhs_tc.cuh")


def _kernels(src):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^{;]*?\)\s*)?(\w+)\(([^{;]*?)\)\s*\{", src):
        yield m.group(1), m.group(2), _body(src, m.start())


def test_every_kernel_that_overlaps_its_predecessor_waits():
    """Each kernel launched with the attribute calls pdl_wait, itself or in its body function."""
    capi = _source("dgtd_capi.cu")
    launched = set(re.findall(r"launch_pdl\((?:dgtd::)?(k_\w+)", capi))
    assert len(launched) >= 15
    bodies = {n: b for f in FILES for n, _, b in _kernels(_source(f))}
    assert launched <= set(bodies)
    for name in launched | {"rhs_tc_kernel"}:
        assert "pdl_wait()" in bodies[name], name
    fp32 = _source("rhs_fp32.cuh")
    for fn in ("rhs_cc_body", "rhs_cc_pair_body"):
        body = _body(fp32, fp32.index("void " + fn + "("))
        assert "pdl_wait()" in body and body.index("pdl_wait()") < body.index("return"), fn


def test_no_read_only_load_of_what_an_earlier_kernel_writes():
    for f in FILES:
        src = _source(f)
        for name, params, body in _kernels(src):
            if "pdl_wait()" not in body and not name.startswith("rhs_"):
                continue
            restricted = set(re.findall(r"__restrict__\s+(\w+)", params + body))
            assert restricted <= HOST_WRITTEN.get(name, set()), (f, name, restricted)
    for f in ("dgtd_common.cuh", "rhs_fp32.cuh", "rhs_tc.cuh"):
        src = _source(f)
        assert "__restrict__" not in src, f
        # element records only (read through m4)
        assert set(re.findall(r"__ldg\(([^()]*)", src)) <= {"m4 + i"}, f
