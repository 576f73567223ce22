"""The bounded waits of the tensor-core CRT lift: one that nothing completes runs
out, records YELL_ERR_TIMEOUT and lets the CTA's next wait return at once; the
status is read and cleared, and lifts afterwards run normally.  A lift of host
limbs has a status word of its own: the one recorded for lifts of device arrays
is neither read nor cleared by it."""
import ctypes
import os
import re
import time

import numpy as np
import pytest

import yell_gb300 as y
from oracle.crt import poly2bigint
from yell_gb300._capi import YELL_ERR_TIMEOUT, call
from yell_gb300.inputs import uniform_polys

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")


def _check(seconds):
    st = ctypes.c_uint32(0)
    call("yell_crt_wait_check", int(seconds * 1e9), ctypes.byref(st))
    return st.value


def _status():
    st = ctypes.c_uint32(99)
    call("yell_crt_wait_status", ctypes.byref(st))
    return st.value


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_reported(cuda):
    assert _check(0.001) == YELL_ERR_TIMEOUT  # loads the kernel
    t0 = time.perf_counter()
    assert _check(0.4) == YELL_ERR_TIMEOUT
    assert 0.4 <= time.perf_counter() - t0 < 0.75  # one wait, not two
    assert _status() == 0
    with pytest.raises(y.YellError):
        _check(0.0)
    for L in (4, 12):
        ps = y.primes(L)
        limbs = [np.ascontiguousarray(l) for l in uniform_polys(5 + L, 1, L, 9, ps)[0]]
        got = y.words_to_ints(y.poly_to_bigint(limbs))
        assert got == poly2bigint(np.stack(limbs), [int(p) for p in ps])
    assert _status() == 0


def test_host_lift_returns_its_own_status():
    """The wait of a real lift cannot be made to run out without a fault, so the
    host call's use of its status is read from the source."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "crt.cu")).read())
    body = text[text.index("int yell_poly_to_bigint("):]
    steps = ["cudaMemsetAsync(d_status, 0", "crt_lift(d_out, d_in, 1, L, log_n, 0, s, ctx->device(), d_status)",
             "take_status(d_status, s, &status)", "return status == kOk ? kOk : fail((int)status"]
    at = [body.index(s) for s in steps]
    assert at == sorted(at)
