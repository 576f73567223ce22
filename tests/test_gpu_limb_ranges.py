"""The ranges of limbs that a variant for few limbs is chosen for: on both
sides of every end, as in test_gpu_few_limbs (whose counts cover the ranges'
upper ends beyond these)."""
import os
import subprocess
import sys

import pytest

from test_gpu_few_limbs import SCRIPT

pytestmark = pytest.mark.gpu

COUNTS = {10: [80, 81, 160, 161, 1024, 1025], 12: [48, 49],
          13: [15, 16, 19, 20, 33, 34, 39, 40, 48, 49, 52, 53, 56], 14: [11, 12, 28, 29, 128, 129, 192, 193],
          15: [4, 5, 14, 15, 96, 97], 16: [2, 3, 7, 10, 11, 64, 65], 17: [2, 3, 5, 64, 65]}


@pytest.mark.parametrize("log_n", sorted(COUNTS))
def test_both_sides_of_the_ranges(cuda, orc, log_n):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "YELL_GB300_TUNE_FILE"}
    r = subprocess.run([sys.executable, "-c", SCRIPT % (log_n, COUNTS[log_n])], cwd=root, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "few limbs ok" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]


TUNED = SCRIPT.replace("digests = {}", "y.autotune(log_n, 1, 2)\ndigests = {}")


@pytest.mark.parametrize("log_n,counts", [(10, [2, 4098]), (13, [16, 1000]), (14, [11, 40, 512]), (16, [2, 8, 200])])
def test_tuned_degree_keeps_the_variants_for_few_limbs(cuda, orc, log_n, counts):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "YELL_GB300_TUNE_FILE"}
    r = subprocess.run([sys.executable, "-c", TUNED % (log_n, counts)], cwd=root, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "few limbs ok" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]
