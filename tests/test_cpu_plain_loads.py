"""Kernels launched as dependents read the caller's words, and those that the
kernel before them leaves in a workspace, by plain loads.  The
read-only path (__ldg, ld.global.nc, const __restrict__) promises that nobody
writes the memory while the kernel runs, and such a kernel is already running,
waiting, beside the kernel that writes its operands; it stays for the library's
own tables.  A stale read cannot be provoked at will, so the sources are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")
TABLES = re.compile(r"mods|cdt|qw|image|\btw\b|m\.fwd|m\.inv|->p\b|->pn\b")


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name", ["ntt_kernels.cuh", "ntt_cluster.cuh", "ntt_dispatch.cu", "ntt32.cu", "crt_mma.cuh",
                                  "samplers.cu"])
def test_read_only_loads_are_of_tables(name):
    for line in _code(name).splitlines():
        if "__ldg(" in line:
            assert TABLES.search(line), (name, line.strip())
        assert "ld.global.nc" not in line and not re.search(r"const uint(32|64)_t\* __restrict__ (a|b|in|src|data)\b", line)
