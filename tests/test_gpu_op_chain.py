"""Chains of whole-limb, cluster and two-pass transforms and element-wise ops,
each launched as a programmatic dependent of the one before and reading its
words: the result is the oracle's, at sizes below, at and above one step of
the element-wise grid."""
import numpy as np
import pytest

import yell_gb300 as y
from yell_gb300.inputs import uniform_polys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,count,L", [(3, 5, 3), (6, 1, 1), (9, 3, 2), (10, 70, 1), (12, 7, 3), (13, 2, 5), (15, 3, 3),
                                           (16, 10, 8)])
def test_chain(cuda, orc, log_n, count, L):
    torch = cuda
    cm0 = 4
    n = 1 << log_n
    ps = y.primes(L, cm0)
    a, b, c = (uniform_polys(40 + k, count, L, log_n, ps) for k in range(3))
    da, db, dc = (torch.from_numpy(v.view(np.int64).copy()).cuda() for v in (a, b, c))
    d = torch.empty_like(da)
    shape = (count, L, log_n, cm0)
    torch.cuda.synchronize()
    y.dev_ntt(da, *shape)
    y.dev_ntt(db, *shape)
    y.dev_elementwise(y.YELL_OP_MULMOD, d, da, db, *shape)
    y.dev_elementwise(y.YELL_OP_ADDMOD, db, d, dc, *shape)
    y.dev_elementwise(y.YELL_OP_MULADD, dc, db, da, *shape)
    y.dev_elementwise(y.YELL_OP_SUBMOD, d, dc, d, *shape)
    y.dev_elementwise(y.YELL_OP_NEGATE, da, d, None, *shape)
    y.dev_elementwise(y.YELL_OP_ADDMOD, da, da, da, *shape)
    y.dev_ntt(da, *shape, y.YELL_BACKWARD)
    torch.cuda.synchronize()
    got = da.cpu().numpy().view(np.uint64).reshape(count, L, n)
    for i, l in {(0, 0), (count // 2, L - 1), (count - 1, 0), (count - 1, L - 1)}:
        cm = cm0 + l
        x, z, w = orc.forward(a[i, l], log_n, cm), orc.forward(b[i, l], log_n, cm), c[i, l]
        m = orc.mulmod(x, z, cm)
        s = orc.addmod(m, w, cm)
        t = orc.negate(orc.submod(orc.muladd(w, s, x, cm), m, cm), cm)
        assert np.array_equal(got[i, l], orc.backward(orc.addmod(t, t, cm), log_n, cm)), (i, l)
