"""Kernels launched by launch_overlapped() (csrc/launch.cuh) start before the
kernel before them has written its results: what an earlier launch may write
must not go through the read-only path.

Reads the sources: the kernels so launched, their parameters (const
__restrict__ lets the compiler take that path) and their __ldg loads.  Allowed
are the tables that the host waits for when a context is built.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "nemo3d_b200", "csrc")
# launch_overlapped's first argument -> the kernel
LAUNCHED = {"kernel": "k_hx_ring", "k_update<VT>": "k_update", "k_clear": "k_clear"}
# written by the build and waited for by the host
FIXED = {"order", "bonds", "onsite", "blocks"}


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            yield name, re.sub(r"//[^\n]*", "", text)


def _kernel(text, name):
    """(parameters, body) of a kernel, by its braces."""
    at = re.search(r"\n\s*%s\(" % name, text) or re.search(r"void %s\(" % name, text)
    open_ = text.index("(", at.start())
    close = open_
    depth = 0
    for k in range(open_, len(text)):
        depth += {"(": 1, ")": -1}.get(text[k], 0)
        if depth == 0:
            close = k
            break
    start = text.index("{", close)
    depth = 0
    for k in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[open_ + 1:close], text[start:k]
    raise AssertionError(name)


def test_overlapped_kernels_read_fresh_values():
    seen = set()
    for name, text in _sources():
        for first in re.findall(r"\blaunch_overlapped\(([^,]+),", text):
            if first.startswith("void"):
                continue  # the definition
            kernel = LAUNCHED[first.strip()]
            seen.add(kernel)
            params, body = _kernel(text, kernel)
            assert "wait_for_previous();" in body, (name, kernel)
            restrict = set(re.findall(r"const [^,]*__restrict__ (\w+)", params))
            assert restrict <= FIXED, (name, kernel, restrict - FIXED)
            through = {re.match(r"\w+", a).group() for a in re.findall(r"__ldg\(([^)]*)\)", body)}
            assert through <= FIXED, (name, kernel, through - FIXED)
    assert seen == set(LAUNCHED.values())
