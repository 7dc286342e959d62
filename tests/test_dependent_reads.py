"""Kernels launched as programmatic dependents are resident while the kernel before them still writes the element
kernels' x and the gathers' R, so they may not read these through the read-only path."""
import glob
import os
import re

from conftest import ROOT


def _functions(text):
    """(header, body) of every device function and kernel of a source file."""
    for m in re.finditer(r"(__global__|__device__)[^;{}]*\{", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(0), text[m.end():end]


def test_no_read_only_loads_of_what_the_kernel_before_writes():
    dependents, readers = 0, 0
    for path in glob.glob(os.path.join(ROOT, "montjoie_gb300", "csrc", "mj_k*")):
        for head, body in _functions(re.sub(r"//.*", "", open(path).read())):
            dependent = "dependent_wait();" in body
            if dependent or re.search(r"contrib_sums_(global|block)\(", head):
                dependents += dependent
                readers += "ld_fresh(" in body
                assert not re.search(r"__ldg\(\s*[xR]\b", body), (path, head)
                assert not re.search(r"\bx\[", body), (path, head)
    assert dependents >= 9 and readers >= 5
