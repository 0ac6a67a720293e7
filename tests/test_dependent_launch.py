"""Kernels launched as programmatic dependents may read mesh data only before
pdl_wait (csrc/kernels.cuh): what stands before it in each of them, and in the
functions called there, names no buffer that a kernel writes."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgm_b200", "csrc")
SOURCES = {os.path.basename(f): open(f).read() for f in glob.glob(os.path.join(CSRC, "*.cuh"))}
WRITTEN = re.compile(r"\ba\.(uref|X|Xn|U|Ut|Utf|A|Tin|Tinf|V|Pv|Ghat|R0)\b|\btrace_in\b")


def body(name):
    for s in SOURCES.values():
        m = re.search(r"__device__ __forceinline__ [\w ]+ " + name + r"\([^;{]*\{.*?\n\}\n", s, re.S)
        if m:
            return m.group(0)
    return ""


def sites():
    for f, s in sorted(SOURCES.items()):
        for k, m in enumerate(re.finditer(r"(?<!void )pdl_wait\(\);", s)):
            yield pytest.param(s[s.rindex("\ntemplate", 0, m.start()):m.start()], id=f"{f}-{k}")


@pytest.mark.parametrize("before", list(sites()))
def test_mesh_data_only_before_the_wait(before):
    assert not WRITTEN.search(before)
    for name in set(re.findall(r"\b(\w+)(?:<[\w:, ]*>)?\(", before)):
        assert not WRITTEN.search(body(name)), name
