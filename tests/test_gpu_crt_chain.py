"""Lifts of few moduli, launched as programmatic dependents: a lift right after
the transform that writes its residues gives the words of the same lift with
the device idle between them."""
import numpy as np
import pytest

import yell_gb300 as y
from yell_gb300.inputs import uniform_polys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,count,L", [(3, 1, 2), (10, 3, 3), (12, 40, 2), (15, 9, 3), (13, 2, 5), (12, 1, 34)])
def test_lift_after_transform(cuda, log_n, count, L):
    torch = cuda
    words = uniform_polys(21, count, L, log_n, y.primes(L))
    W = y.crt_words(L)

    def run(between):
        x = torch.from_numpy(words.view(np.int64).copy()).cuda()
        out = torch.empty((count << log_n) * W, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):
            y.dev_ntt(x, count, L, log_n, 0, y.YELL_BACKWARD)
            if between:
                torch.cuda.synchronize()
            y.dev_crt_lift(out, x, count, L, log_n)
            if between:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return out

    assert torch.equal(run(False), run(True))
