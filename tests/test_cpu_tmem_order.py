"""Where the tensor-core CRT kernel takes tensor memory: after the wait for the
stream's previous kernel and before it lets the next one start.  A CTA holding
TMEM columns while it waits, or one whose dependents may already hold them,
could wait for ever for a kernel that allocates TMEM too; that cannot be shown
on a GPU without hanging it, so the order is read from the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")


def test_allocation_between_wait_and_launch():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "crt_mma.cuh")).read())
    body = text[text.index("k_crt_mma("):]
    steps = ["grid_dep_wait()", "tcgen05.alloc", "tmem_address(bars)", "grid_dep_launch()", "tcgen05.dealloc"]
    at = [body.index(s) for s in steps]
    assert at == sorted(at), dict(zip(steps, at))
    assert all(body.count(s) == 1 for s in ("grid_dep_wait()", "tcgen05.alloc", "grid_dep_launch()"))
