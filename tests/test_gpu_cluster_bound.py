"""Where the device cannot place clusters of 8, 4 or 2 CTAs (a small partition;
here YELL_GB300_MAX_CLUSTER), calls take kernels that it can place, with the
oracle's words.  In processes of their own: the bound is read once per device."""
import os
import subprocess
import sys

import pytest

from test_gpu_few_limbs import SCRIPT

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(args, bound):
    env = {k: v for k, v in os.environ.items() if k != "YELL_GB300_TUNE_FILE"}
    r = subprocess.run([sys.executable, *args], cwd=ROOT, env=dict(env, YELL_GB300_MAX_CLUSTER=str(bound)),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-1500:] + r.stderr[-1500:]
    return r.stdout


@pytest.mark.parametrize("log_n,bound", [(10, 2), (11, 2), (12, 4), (13, 4), (13, 1), (14, 4)])
def test_64_bit_calls(cuda, orc, log_n, bound):
    script = SCRIPT % (log_n, [1, 11]) + r"""
import re
names = y.variants(log_n)
for limbs in (1, 11, 60, 1000):
    for polymul in (False, True):
        m = re.match("cluster of ([0-9]+)", names[y.variant_for(log_n, limbs, polymul)])
        assert not m or int(m[1]) <= int(__import__("os").environ["YELL_GB300_MAX_CLUSTER"]), (limbs, m)
print("bound ok")
"""
    out = _run(["-c", script], bound)
    assert "few limbs ok" in out and "bound ok" in out


@pytest.mark.parametrize("bound,degrees", [(4, "13 or 14 or 15"), (2, "12 or 13 or 14 or 15"), (1, "10 or 12 or 13")])
def test_32_bit_calls(cuda, bound, degrees):
    out = _run(["-m", "pytest", "-q", "-m", "gpu", "tests/test_gpu_ntt32_routes.py", "-k", degrees], bound)
    assert "passed" in out and "failed" not in out


def test_32_bit_degrees_that_need_a_cluster(cuda):
    """2^14 and 2^15 need clusters of 2: without them a call is an error."""
    script = r"""
import torch
from yell_gb300 import moduli32 as m32, YellError
t = torch.zeros(1 << 14, dtype=torch.int32, device="cuda")
try:
    m32.dev_ntt(t, 1, 1, 14)
except YellError as e:
    print("refused", e)
torch.cuda.synchronize()
"""
    assert "refused" in _run(["-c", script], 1)
