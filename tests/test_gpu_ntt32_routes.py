"""32-bit transforms and polymul on both sides of every number of limbs at
which another kernel takes over (clusters of 2, 4 and 8 CTAs, the staged CTA
pair, one CTA per limb): the oracle's words.  Limbs repeat with period two, so
that every limb of a call is compared."""
import numpy as np
import pytest

import oracle
from yell_gb300 import moduli32 as m32
from yell_gb300.inputs import splitmix64

pytestmark = pytest.mark.gpu

COUNTS = {10: [1, 1024, 1025], 11: [1, 512, 513, 768, 769, 1024, 1025], 12: [1, 224, 225, 288, 289, 768, 769, 1536, 1537],
          13: [1, 100, 101, 400, 401, 768, 769], 14: [1, 76, 77, 200, 201], 15: [1, 32, 33, 57, 58, 76, 77]}


@pytest.mark.parametrize("log_n", sorted(COUNTS))
def test_both_sides_of_the_bounds(cuda, log_n):
    torch = cuda
    orc = oracle.Oracle32("port")
    n, cm0 = 1 << log_n, 5
    p = np.array([m32.prime(cm0), m32.prime(cm0 + 1)], dtype=np.uint64).reshape(2, 1)
    # words below 4p for the forward transforms, below 2p for the inverse, reduced operands
    x4 = (splitmix64(log_n, 2 * n).reshape(2, n) % (4 * p)).astype(np.uint32)
    x2, a = (x4 % (2 * p)).astype(np.uint32), (x4 % p).astype(np.uint32)
    b = (splitmix64(log_n + 100, 2 * n).reshape(2, n) % p).astype(np.uint32)
    want = {"polymul": [orc.polymul(a[l][None], b[l][None], log_n, cm0 + l)[0] for l in range(2)]}
    for name, x in (("forward", x4), ("forward_lazy", x4), ("backward", x2)):
        want[name] = [getattr(orc, name)(x[l], log_n, cm0 + l) for l in range(2)]

    def dev(words, count):
        t = torch.from_numpy(words.view(np.int32).copy()).cuda()
        return t.repeat((count + 1) // 2, 1)[:count].contiguous()

    def check(t, name, count, L):
        got = t.cpu().numpy().view(np.uint32).reshape(count, n)
        for i in range(count):
            assert np.array_equal(got[i], want[name][i % L]), (name, count, i)

    for count in COUNTS[log_n]:
        L = 2 if count % 2 == 0 else 1
        rows = slice(0, L)
        for direction, name, x in ((m32.YELL_FORWARD, "forward", x4), (m32.YELL_FORWARD_LAZY, "forward_lazy", x4),
                                   (m32.YELL_BACKWARD, "backward", x2)):
            t = dev(x if L == 2 else np.repeat(x[rows], 2, axis=0), count)
            torch.cuda.synchronize()
            m32.dev_ntt(t, count // L, L, log_n, cm0, direction)
            torch.cuda.synchronize()
            check(t, name, count, L)
        da, db = (dev(w if L == 2 else np.repeat(w[rows], 2, axis=0), count) for w in (a, b))
        c = torch.zeros_like(da)
        torch.cuda.synchronize()
        m32.dev_polymul(c, da, db, count // L, L, log_n, cm0)
        torch.cuda.synchronize()
        check(c, "polymul", count, L)
    assert m32.wait_status() == 0
