"""Chains of 32-bit transforms, polymuls and element-wise ops, each launched as
a programmatic dependent of the one before and reading its words: the words
are those of the same calls with the device idle between them."""
import numpy as np
import pytest

import yell_gb300 as y
from yell_gb300 import moduli32 as m32
from yell_gb300.inputs import splitmix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,count,L", [(3, 5, 3), (7, 40, 2), (9, 700, 1), (10, 1100, 1), (12, 3, 2), (13, 9, 5), (15, 3, 2)])
def test_chain(cuda, log_n, count, L):
    torch = cuda
    cm0, n = 2, 1 << log_n
    p = np.array([m32.prime(cm0 + l) for l in range(L)], dtype=np.uint64).reshape(1, L, 1)
    words = [(splitmix64(90 + k, count * L * n).reshape(count, L, n) % p).astype(np.uint32).view(np.int32) for k in range(2)]
    shape = (count, L, log_n, cm0)

    def run(between):
        a, b = (torch.from_numpy(w.copy()).cuda().reshape(-1) for w in words)
        c, d = torch.empty_like(a), torch.empty_like(a)
        torch.cuda.synchronize()
        for f in (lambda: m32.dev_ntt(a, *shape), lambda: m32.dev_ntt(b, *shape),
                  lambda: m32.dev_elementwise(y.YELL_OP_MULMOD, c, a, b, *shape),
                  lambda: m32.dev_ntt(c, *shape, y.YELL_BACKWARD), lambda: m32.dev_polymul(d, c, b, *shape),
                  lambda: m32.dev_elementwise(y.YELL_OP_ADDMOD, a, d, c, *shape),
                  lambda: m32.dev_ntt(a, *shape, y.YELL_FORWARD_LAZY)):
            f()
            if between:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return a, c, d

    for _ in range(3):
        for x, z in zip(run(False), run(True)):
            assert torch.equal(x, z)
