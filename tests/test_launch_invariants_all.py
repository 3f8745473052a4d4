"""The rule of dependent launches (wait first, once) over every CUDA source, and
over both launch helpers (CPU, reads the sources).

A kernel launched with `launch_k` or `launch_on` calls `pdl_entry()` exactly once,
with no return and no store through its pointer parameters before it; nothing but
a kernel calls it, since a helper's wait would run wherever the helper is used.
"""
import glob
import os
import re

import pytest

from test_launch_invariants import CSRC, _bodies, _violations


def _all_sources():
    return {os.path.basename(f): open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def _launched(srcs):
    names = set()
    for s in srcs.values():
        names |= set(re.findall(r"\blaunch_k\(c,\s*([A-Za-z_0-9]+)", s))
        names |= set(re.findall(r"\blaunch_on\(c,\s*st,\s*([A-Za-z_0-9]+)", s))
    return sorted(names)


def _outside(srcs):
    """Calls of pdl_entry() that lie in no kernel, as file:line."""
    out = []
    for f, s in srcs.items():
        inside = set()
        for m in re.finditer(r"__global__", s):
            brace, semi = s.find("{", m.end()), s.find(";", m.end())
            if 0 <= brace < semi:  # else a declaration
                inside |= set(range(brace, s.index("\n}\n", brace)))
        out += [f"{f}:{s[:m.start()].count(chr(10)) + 1}" for m in re.finditer(r"\bpdl_entry\(\);", s)
                if m.start() not in inside]
    return out


def test_every_launch_is_seen():
    """No launch through a helper escapes the two patterns above."""
    srcs = _all_sources()
    for f, s in srcs.items():
        calls = len(re.findall(r"\blaunch_(?:k|on)\((?!const)", s))
        seen = len(re.findall(r"\blaunch_(?:k\(c,|on\(c,\s*st,)\s*k[A-Za-z_0-9]*", s))
        assert calls - seen == (1 if f == "mac_internal.cuh" else 0), f  # launch_k is one call of launch_on
    assert len(_launched(srcs)) >= 70


@pytest.mark.parametrize("name", _launched(_all_sources()))
def test_dependent_launch_kernel_waits_first(name):
    bodies = _bodies(_all_sources(), name)
    assert bodies, name
    for params, body in bodies:
        assert _violations(name, params, body) == []


def test_nothing_but_kernels_waits():
    assert _outside(_all_sources()) == []


def test_checker_flags_a_planted_helper():
    helper = "__device__ int f() {\n  pdl_entry();\n  return 1;\n}\n"
    kernel = "__global__ void k(int* a) {\n  pdl_entry();\n  a[0] = f();\n}\n"
    assert _outside({"x.cu": kernel}) == []
    assert _outside({"x.cu": kernel + helper}) == ["x.cu:6"]
