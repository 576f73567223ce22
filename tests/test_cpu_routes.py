"""Which variant a call of so many limbs takes: the rule (of the ranges that
hold the number the one that ends first, else the degree's first variant, at
2^13 two passes at k1 = 6), applied here to the ranges as the sources register
them, on both sides of every end."""
import os
import re

import pytest

import yell_gb300 as y

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")
ANY = (1 << 32) - 1
FILES = ("ntt_whole_few.cu", "ntt_two_pass_few.cu", "ntt_cluster.cu")  # in the order of registration


def registered():
    """{log_n: [(polymul ranges, transform ranges)]} in the order of registration."""
    out = {}
    number = lambda s: ANY if s == "kAnyLimbs" else int(s)  # noqa: E731
    for name in FILES:
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        calls = re.findall(r"by\[(\d+)\]\.push_back\(upto\(\w+<[^>]*>\(\), (\w+), (\w+)((?:, \{[^}]*\})*)\)\);", text)
        assert len(calls) == text.count("push_back")
        for degree, polymul, ntt, more in calls:
            also = [tuple(number(v) for v in re.findall(r"\d+", r)) for r in re.findall(r"\{([^}]*)\}", more)]
            also += [()] * (2 - len(also))
            out.setdefault(int(degree), []).append(
                tuple([r for r in ((1, number(first)), further) if r and r[0] <= r[1]]
                      for first, further in ((polymul, also[0]), (ntt, also[1]))))
    return out


def ends(log_n):
    """Numbers of limbs at and next to every end of the degree's ranges."""
    at = set()
    for kinds in registered().get(log_n, []):
        for least, most in kinds[0] + kinds[1]:
            at |= {n for e in (least, most) if e != ANY for n in (e - 1, e, e + 1) if n > 0}
    return sorted(at)


def test_every_degree_with_ranges_is_seen():
    assert sorted(registered()) == [6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20]


@pytest.mark.parametrize("log_n", range(3, 21))
def test_the_picked_variant(ylib, log_n):
    few = registered().get(log_n, [])
    names = y.variants(log_n)
    first = len(names) - 1 - len(few)  # the last variant is the first one again
    assert names[-1].startswith(names[0]) and first >= 1
    for limbs in ends(log_n) + [1, 2, 100000]:
        for kind, polymul in ((0, True), (1, False)):
            held = [(most, first + k) for k, kinds in enumerate(few)
                    for least, most in kinds[kind] if least <= limbs <= most]
            want = min(held)[1] if held else (1 if log_n == 13 else 0)
            assert y.variant_for(log_n, limbs, polymul) == want, (limbs, polymul)
    if few:
        assert y.variant_for(log_n, 1, True) >= first
