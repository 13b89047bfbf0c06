"""The kernels' bounded waits, from the source: each tells the host or its caller
that it ran out, and what a kernel then still writes as an index is in range. (On a
GPU a wait only runs out when something is broken.)"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flowpanel.jl_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


def functions(path):
    """(signature, body) of every function of a source file, comments removed."""
    src = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__(?:device|global)__[^;{}=]*?\)\s*\{", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(0), src[m.end():i]


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_every_wait_reports(path):
    for head, body in functions(path):
        if re.search(r"try_wait\.parity|\b(kSpin|kSpinLimit|kWaitLimit)\b", body):
            assert "DEV_TIMEOUT" in body or re.search(r"\bbool\s+mbar_\w+\(|\bint& late\)", head), head
        if "wait_step(" in body:   # its expiry is kept in `late` until the warp's last wait
            assert "step_status(late, status)" in body[body.rindex("wait_step("):], head


def test_panel_row_order_is_set_before_any_wait():
    body = next(b for h, b in functions(os.path.join(CSRC, "fp_lu64.cu")) if "k_panel64(" in h)
    order = body.index("s.pr[tid] = s.lp[tid] = tid")
    assert order < body.index("wait_flag") and order < body.index("diagonal()") and order < body.index("rest()")
