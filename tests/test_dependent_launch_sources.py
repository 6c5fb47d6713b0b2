"""Kernels that may start before the kernel in front of them has ended.

They read memory that the earlier kernel still writes, behind their own wait.  A
parameter that is `const` and `__restrict__` promises the compiler memory that nobody
writes during the kernel (it may then read through the non-coherent path and move the
reads), which is not so for them.
"""
from __future__ import annotations

import os
import re


CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ncsim_b200", "csrc")
WAITS = re.compile(r"after_previous_kernel\(\);|griddepcontrol\.wait")


def _kernels(path):
    """(name, parameters) of every kernel that waits for the kernel before it."""
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for part in text.split("__global__")[1:]:
        head, body = part[: part.index("{")], part[part.index("{") :]
        body = re.split(r"\n}", body, maxsplit=1)[0]  # up to the kernel's closing brace
        if WAITS.search(body):
            head = re.sub(r"__launch_bounds__\([^)]*\)", "", head)
            yield head.split("(")[0].split()[-1], head[head.index("(") + 1 :]


def test_kernels_that_wait_promise_nothing_about_memory_in_flight():
    found = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            found.update({k: p for k, p in _kernels(os.path.join(CSRC, name))})
    # the measurement's kernels, the tiled pass and the fused pass
    assert {"k_expect_diag", "k_expect_pair", "k_project_diag", "k_project_pair", "k_flip_if", "k_plain_pass", "k_fused_pass"} <= set(found)
    bad = [k for k, p in found.items() if any("const" in q.split("*")[0] and "__restrict__" in q for q in p.split(","))]
    assert not bad, bad
