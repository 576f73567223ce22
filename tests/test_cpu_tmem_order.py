"""Where the tensor-core CRT kernel takes tensor memory: after the wait for the
stream's previous kernel, before it lets the next one start, and before any of
its bounded waits.  A CTA holding TMEM columns while it waits, or one whose
dependents may already hold them, could wait for ever for a kernel that
allocates TMEM too; that cannot be shown on a GPU without hanging it, so the
order is read from the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")


def _kernel():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "crt_mma.cuh")).read())
    return text[text.index("k_crt_mma("):]


def test_allocation_between_wait_and_launch():
    body = _kernel()
    assert all(body.count(s) == 1 for s in ("grid_dep_wait()", "tcgen05.alloc", "grid_dep_launch()", "tcgen05.dealloc"))
    wait, alloc, launch = (body.index(s) for s in ("grid_dep_wait()", "tcgen05.alloc", "grid_dep_launch()"))
    assert wait < alloc < body.index("tmem_address(bars)", alloc) < launch < body.index("tcgen05.dealloc")


def test_every_role_meets_after_the_allocation_before_it_waits():
    body = _kernel()
    roles = body[body.index("if (warp >= kEpilogueWarps &&"):]
    roles = re.split(r"\n  \} else (?:if \(warp == [^\n]*\) )?\{\n", roles)
    assert len(roles) == 3  # producers, issuing warp, epilogue
    for role in roles:
        assert role.count("tmem_address(bars)") == 1
        assert role.index("tmem_address(bars)") < role.index("wait(bars,")
