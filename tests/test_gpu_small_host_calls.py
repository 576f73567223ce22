"""Small host calls run in place on the mapped host buffer when the dispatch
makes them one launch, whatever variant the tuner chose for larger calls: they
reserve no device staging.  In a process of its own, with two passes as the
tuner's choice at 2^13."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import numpy as np
import yell_gb300 as y
from oracle import Oracle
from yell_gb300.inputs import uniform_polys
orc = Oracle("port")
log_n = 13
names = y.variants(log_n)
assert names[y.get_variant(log_n)].startswith("two-pass") and "tiles of" not in names[y.get_variant(log_n)]
y.poly_forward([np.zeros(16, np.uint64)])  # brings the mapped buffer up
for L in (1, 2, 4):
    ps = y.primes(L)
    a, b = (uniform_polys(k, 1, L, log_n, ps) for k in (L, L + 9))
    y.init_ntt_tables(log_n, L)
    before = y.allocations()
    got = y.polymul_host(a, b, log_n)
    limbs = [l.copy() for l in a[0]]
    y.poly_forward(limbs)
    assert y.allocations() == before, L
    assert np.array_equal(got[0], orc.polymul(a[0], b[0], log_n, 0))
    assert all(np.array_equal(limbs[l], orc.forward(a[0, l], log_n, l)) for l in range(L))
print("small host calls ok")
"""


def test_small_calls_after_tuning(cuda, orc, tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    tune = tmp_path / "tune"
    tune.write_text(f"{cuda.cuda.get_device_name(0)}|13|two-pass k1=6 (columns of 2^6, rows of 2^7)\n")
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, env=dict(os.environ, YELL_GB300_TUNE_FILE=str(tune)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "small host calls ok" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]
