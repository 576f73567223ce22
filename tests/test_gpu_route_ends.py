"""On both sides of every end of the ranges of limbs that variants are
registered for, at every degree: the words of the variant that the call takes
are those of the degree's first variant at every limb, and at the first and the
last limb the oracle's.  In a process of its own per degree: a selection made
by another test would hold."""
import os
import subprocess
import sys

import pytest

from test_cpu_routes import ends, registered

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import numpy as np, torch
import yell_gb300 as y
from oracle import Oracle
orc = Oracle("port")
log_n, counts, cm0 = %d, %r, 3
n, last = 1 << log_n, len(y.variants(log_n)) - 1
p = [y.prime(cm0), y.prime(cm0 + 1)]
g = torch.Generator(device="cuda")
g.manual_seed(log_n)

def run(a, b, count, L):
    out = [torch.empty_like(a)]
    y.dev_polymul(out[0], a, b, count // L, L, log_n, cm0)
    for direction in (0, 1, 2):
        out.append(a.clone())
        torch.cuda.synchronize()
        y.dev_ntt(out[-1], count // L, L, log_n, cm0, direction)
    torch.cuda.synchronize()
    return out

for count in counts:
    L = 2 if count %% 2 == 0 else 1
    a, b = (torch.randint(0, min(p), (count, n), generator=g, device="cuda", dtype=torch.int64) for _ in range(2))
    torch.cuda.synchronize()
    y.set_variant(log_n, 0)
    got = run(a, b, count, L)
    picked = {y.variant_for(log_n, count, k) for k in (False, True)}
    y.set_variant(log_n, last)
    assert y.variant_for(log_n, count) == last and picked != {last}
    want = run(a, b, count, L)
    assert all(torch.equal(x, z) for x, z in zip(got, want)), count
    for i in (0, count - 1):
        cm = cm0 + (L - 1 if i else 0)
        x, z, *w = (t[i].cpu().numpy().view(np.uint64) for t in (a, b, *got))
        assert np.array_equal(w[0], orc.polymul(x[None], z[None], log_n, cm)[0]), (count, i)
        for f, v in zip((orc.forward, orc.forward_lazy, orc.backward), w[1:]):
            assert np.array_equal(v, f(x, log_n, cm)), (count, i, f.__name__)
print("route ends ok")
"""


@pytest.mark.parametrize("log_n", sorted(registered()))
def test_both_sides_of_every_end(cuda, orc, log_n):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "YELL_GB300_TUNE_FILE"}
    r = subprocess.run([sys.executable, "-c", SCRIPT % (log_n, ends(log_n))], cwd=root, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "route ends ok" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]
