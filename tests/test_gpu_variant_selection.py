"""Selecting a variant and selecting the earlier one again leaves a degree's
dispatch as it was, whether nothing, the autotuner's choice or a variant by hand
was selected before: shown by the number of kernels that calls launch and by the
variant they report."""
import pytest

import yell_gb300 as y

pytestmark = pytest.mark.gpu

# limbs of calls that take a cluster or small tiles, or the variant for all others
LIMBS = {10: (1, 200, 5000), 13: (1, 18, 400, 1000), 14: (1, 20, 100, 600), 16: (1, 9, 50, 300)}


def _routes(torch, log_n):
    """Per number of limbs and kind: the variant, and the kernels launched (transforms of up to 20 limbs)."""
    out = []
    for limbs in LIMBS[log_n]:
        for polymul in (False, True):
            out.append(y.variant_for(log_n, limbs, polymul))
        if limbs <= 20:
            t = torch.zeros(limbs << log_n, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            before = y.kernel_launches()
            y.dev_ntt(t, limbs, 1, log_n)
            out.append(("launches", y.kernel_launches() - before))
            torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("log_n", sorted(LIMBS))
def test_selecting_and_going_back(cuda, log_n):
    torch = cuda
    names = y.variants(log_n)
    y.init_ntt_tables(log_n, 1)
    last = len(names) - 1
    try:
        y.set_variant(log_n, 0)
        assert y.get_variant(log_n) == 0
        default = _routes(torch, log_n)
        assert len(set(r for r in default if not isinstance(r, tuple))) > 1
        for v in (1, last):
            before = y.get_variant(log_n)
            y.set_variant(log_n, v)
            assert y.get_variant(log_n) == v
            assert all(r == v for r in _routes(torch, log_n) if not isinstance(r, tuple))
            y.set_variant(log_n, before)
            assert y.get_variant(log_n) == before and _routes(torch, log_n) == default
        # the last variant is the first one, at every number of limbs
        assert names[last].startswith(names[0])
        # a variant by hand, another, and the first again
        y.set_variant(log_n, 1)
        pinned, before = _routes(torch, log_n), y.get_variant(log_n)
        y.set_variant(log_n, last)
        y.set_variant(log_n, before)
        assert _routes(torch, log_n) == pinned
        # the tuner's choice, another, and the tuner's again
        best, _ = y.autotune(log_n, 2, 2)
        tuned = _routes(torch, log_n)
        assert any(r not in (best, last) for r in tuned if not isinstance(r, tuple))  # few limbs keep theirs
        before = y.get_variant(log_n)
        assert before == best
        y.set_variant(log_n, last)
        y.set_variant(log_n, before)
        assert y.get_variant(log_n) == best and _routes(torch, log_n) == tuned
    finally:
        y.set_variant(log_n, 0)


def test_the_last_variant_runs_the_first_ones_kernels(cuda):
    torch = cuda
    log_n = 14
    t = torch.zeros(1 << log_n, dtype=torch.int64, device="cuda")
    y.init_ntt_tables(log_n, 1)
    torch.cuda.synchronize()
    try:
        y.set_variant(log_n, len(y.variants(log_n)) - 1)
        before = y.kernel_launches()
        y.dev_ntt(t, 1, 1, log_n)
        assert y.kernel_launches() - before == 2  # two passes, where the default is one cluster launch
        torch.cuda.synchronize()
    finally:
        y.set_variant(log_n, 0)
