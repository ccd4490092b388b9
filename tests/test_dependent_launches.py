"""Kernels that may start before the one ahead has ended (they call
wait_for_prior_kernel): that call is their first statement that touches memory, and
only arrays that none of these kernels writes may be declared __restrict__ or read
through the read-only path -- the others change while the kernel is resident.
CPU: reads the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opengraph_b200", "csrc")

# arrays of the graph and of its layouts, complete before the first such launch;
# ctl of spmv_pull_kernel: class counts, written when the graph's rows are classed
CONSTANT = {"lay", "chunks", "vfirst", "vcount", "rows", "rows_f", "rows_i", "nbr", "nbr_f", "nbr_i", "off_light",
            "unit_first", "med_off", "med_v", "out_degree", "perm", "heavy", "light", "med"}
EXTRA = {"spmv_pull_kernel": {"ctl"}}


def text(name):
    t = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", t)


def kernels():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        t = text(f)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\s*\(([^{;]*)\)\s*\{", t):
            end = t.find("\n}\n", m.end())
            body = t[m.end():end]
            if "wait_for_prior_kernel()" in body:
                out.append((f, m.group(1), m.group(2), body))
    return out


KERNELS = kernels()


def test_found():
    assert {k[1] for k in KERNELS} == {"pr_pull_kernel", "pprk_iter", "pprk_check", "msk_expand", "msk_push_long", "msk_finish",
                                       "spmv_pull_kernel", "onesweep_kernel"}


@pytest.mark.parametrize("kernel", KERNELS, ids=[k[1] for k in KERNELS])
def test_only_constant_arrays_are_restrict(kernel):
    _, name, params, body = kernel
    restrict = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert restrict <= CONSTANT | EXTRA.get(name, set()), restrict - CONSTANT
    before = body[:body.index("wait_for_prior_kernel()")]
    # declarations only: shared arrays and constants
    for s in filter(None, (x.strip() for x in before.split(";"))):
        assert re.match(r"(extern\s+)?__shared__|constexpr", s), s
    read = set(re.findall(r"__ldg\(\s*&?(\w+)", body))
    assert read <= CONSTANT, read - CONSTANT


@pytest.mark.parametrize("file,name", [("pagerank.cu", "strided_sum"), ("pagerank.cu", "gather"), ("batch.cu", "ppr_row_sum"),
                                       ("batch.cu", "ms_push4"), ("batch.cu", "ppr_update")])
def test_their_helpers(file, name):
    t = text(file)
    m = re.search(r"__forceinline__\s+\w+\s+%s\s*\(([^{;]*)\)\s*\{" % name, t)
    assert set(re.findall(r"__restrict__\s+(\w+)", m.group(1))) <= CONSTANT
    body = t[m.end():t.index("\n}" if name != "gather" else "\n  }", m.end())]
    assert set(re.findall(r"__ldg\(\s*&?(\w+)", body)) <= CONSTANT
