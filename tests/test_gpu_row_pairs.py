"""Row passes that take the polynomials of a call two at a time: on both sides
of their rules (even, few and many odd polynomials, calls below and above the
inverse's least size, rows of 2^6 to 2^12 words) a call's words are those of
one call per polynomial and, at the first and last limbs, the oracle's."""
import numpy as np
import pytest

import yell_gb300 as y
from yell_gb300.inputs import uniform_polys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,polys,L", [
    (13, 2, 3), (13, 64, 4), (13, 63, 4), (13, 65, 4), (14, 16, 8), (14, 17, 8), (14, 15, 9), (15, 9, 8), (15, 32, 2),
    (16, 3, 11), (16, 2, 16), (16, 17, 2), (17, 2, 8), (18, 4, 2), (19, 2, 2), (20, 2, 1)])
def test_pairs(cuda, orc, log_n, polys, L):
    torch = cuda
    cm0, n = 2, 1 << log_n
    a = uniform_polys(log_n + polys, polys, L, log_n, y.primes(L, cm0))
    src = torch.from_numpy(a.view(np.int64).copy()).cuda()
    ends = {(0, 0), (0, L - 1), (polys - 1, 0), (polys - 1, L - 1)}
    rows = [v for v, name in enumerate(y.variants(log_n)) if name.startswith("two-pass") and "tiles of" not in name]
    try:
        for v in rows:
            y.set_variant(log_n, v)
            for direction in (y.YELL_FORWARD, y.YELL_FORWARD_LAZY, y.YELL_BACKWARD):
                got, one = src.clone(), src.clone().reshape(polys, L * n)
                torch.cuda.synchronize()
                y.dev_ntt(got, polys, L, log_n, cm0, direction)
                for i in range(polys):
                    y.dev_ntt(one[i], 1, L, log_n, cm0, direction)
                torch.cuda.synchronize()
                assert torch.equal(got.reshape(-1), one.reshape(-1)), (v, direction)
                if v == rows[0] and direction != y.YELL_FORWARD_LAZY:
                    words = got.cpu().numpy().view(np.uint64).reshape(polys, L, n)
                    call = orc.forward if direction == y.YELL_FORWARD else orc.backward
                    for i, l in ends:
                        assert np.array_equal(words[i, l], call(a[i, l], log_n, cm0 + l)), (direction, i, l)
    finally:
        y.set_variant(log_n, 0)
