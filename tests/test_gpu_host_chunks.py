"""polymul_host at the edges of its chunks: a single chunk, last chunks of
4 MiB per operand, a remainder, and 64 MiB of operands, where full
chunks come first; pinned and pageable operands."""
import numpy as np
import pytest

import yell_gb300 as y
from yell_gb300.inputs import uniform_polys

pytestmark = pytest.mark.gpu


# a pair of 8 x 2^14 words is 1 MiB: four make a last chunk, 32 a full one
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("pairs", [1, 4, 5, 11, 32, 37])
def test_chunk_edges(cuda, orc, pairs, pinned):
    torch = cuda
    log_n, L = 14, 8
    ps = y.primes(L)
    words = [uniform_polys(70 + k, pairs, L, log_n, ps).view(np.int64) for k in range(2)]
    host = [torch.from_numpy(w) for w in words + [np.zeros_like(words[0])]]
    if pinned:
        host = [h.pin_memory() for h in host]
    a, b, c = (h.numpy().view(np.uint64) for h in host)
    y.polymul_host(a, b, log_n, out=c)
    for i in {0, pairs // 2, pairs - 1}:
        assert np.array_equal(c[i], orc.polymul(a[i], b[i], log_n, 0)), i
    # every pair against the call on device memory
    d = torch.empty_like(host[2], device="cuda")
    y.dev_polymul(d, host[0].cuda(), host[1].cuda(), pairs, L, log_n, 0)
    torch.cuda.synchronize()
    assert np.array_equal(c, d.cpu().numpy().view(np.uint64))
