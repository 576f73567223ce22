"""Calls for which no variant was selected run the variant registered for
their number of limbs (clusters, small tiles, one limb per CTA); on both
sides of every bound the words are those of variant 0 and, for the first and
the last limb, the oracle's.  In a process of its own: a selection made by
another test would hold."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import hashlib
import numpy as np, torch
import yell_gb300 as y
from oracle import Oracle
from yell_gb300.inputs import splitmix64
orc = Oracle("port")
log_n, counts, cm0 = %d, %r, 3
n = 1 << log_n
p = np.array([y.prime(cm0), y.prime(cm0 + 1)], dtype=np.uint64)

def operands(count):
    L = 2 if count %% 2 == 0 else 1
    return L, [w %% p[:L].reshape(1, L, 1) for w in splitmix64(count, 2 * count * n).reshape(2, count // L, L, n)]

def run(count):
    L, (a, b) = operands(count)
    dev = lambda w: torch.from_numpy(w.view(np.int64).copy()).cuda()
    out = [torch.empty(a.size, dtype=torch.int64, device="cuda")]
    y.dev_polymul(out[0], dev(a), dev(b), count // L, L, log_n, cm0)
    for direction in (0, 1, 2):
        out.append(dev(a))
        y.dev_ntt(out[-1], count // L, L, log_n, cm0, direction)
    torch.cuda.synchronize()
    return [t.cpu().numpy().view(np.uint64).reshape(count, n) for t in out]

digests = {}
for count in counts:
    L, (a, b) = operands(count)
    got = run(count)
    for i in (0, -1):
        x, z, cm = a.reshape(count, n)[i], b.reshape(count, n)[i], cm0 + (0 if i == 0 else L - 1)
        assert np.array_equal(got[0][i], orc.polymul(x[None], z[None], log_n, cm)[0]), (count, "polymul")
        for f, w in zip((orc.forward, orc.forward_lazy, orc.backward), got[1:]):
            assert np.array_equal(w[i], f(x, log_n, cm)), (count, f.__name__)
    digests[count] = [hashlib.sha256(w).digest() for w in got]
y.set_variant(log_n, 0)
for count in counts:
    assert digests[count] == [hashlib.sha256(w).digest() for w in run(count)], count
print("few limbs ok")
"""

# 1 limb, and both sides of each bound of the degree
COUNTS = {6: [1, 4096, 4097], 9: [1, 4096, 4097], 10: [1, 48, 49, 256, 257, 384, 385], 11: [1, 7, 1024, 1025],
          12: [1, 12, 13, 160, 161, 640, 641], 13: [1, 12, 13, 32, 33, 64, 65, 320, 321, 768, 769],
          14: [1, 12, 13, 40, 41, 56, 57, 160, 161, 224, 225], 15: [1, 22, 23, 32, 33, 64, 65, 112, 113],
          16: [1, 8, 9, 16, 17, 28, 29, 192, 193], 17: [1, 6, 7, 8, 9, 12, 13, 96, 97], 18: [1, 8, 9, 32, 33],
          20: [1, 4, 5, 12, 13]}


@pytest.mark.parametrize("log_n", sorted(COUNTS))
def test_both_sides_of_the_bounds(cuda, orc, log_n):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "YELL_GB300_TUNE_FILE"}
    r = subprocess.run([sys.executable, "-c", SCRIPT % (log_n, COUNTS[log_n])], cwd=root, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "few limbs ok" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]
