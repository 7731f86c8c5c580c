"""Kernels launched as programmatic successors (CPU only, reads the sources).

Such a kernel starts while the one before it still writes, and waits in its
first statement.  `__restrict__` (with const: read-only for the kernel's
whole life) would let the compiler load above that wait, so only the series
and the training samples, which no kernel writes, may carry it.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paddi_b200", "csrc")
READ_ONLY = {"x", "X", "Yt", "perm"}


def _kernels():
    for fn in sorted(os.listdir(CSRC)):
        if not fn.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, fn)).read())
        for m in re.finditer(r"__global__\s+void\s*(?:__launch_bounds__\s*\([^()]*\)\s*)?(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            body = text[i:text.find("\n}", i)]
            yield fn, m.group(1), text[m.end():i - 1], body


def test_chained_kernels_promise_nothing_about_arrays_that_kernels_write():
    chained = 0
    for fn, name, params, body in _kernels():
        if not re.search(r"\b(chain_begin|st_begin)\(", body):
            continue
        chained += 1
        for p in params.split(","):
            if "__restrict__" in p:
                assert p.split()[-1].lstrip("*") in READ_ONLY, (fn, name, p.strip())
    assert chained >= 18
