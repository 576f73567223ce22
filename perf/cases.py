"""The work whose speed is watched: calls that programs make of this library, over the ranges they use.

`listed()` are the cases that are always timed, `draw(rng)` gives others of the same ranges;
`prepare` makes what a program has in hand before a call (operands on the device, resident
twiddle tables, caller-owned scratch), and `run` is one pass through the public entry points.
Device calls go to the library's own stream (`stream=None`), as most callers leave it.
"""
import numpy as np
import torch

import yell_gb300 as y
from yell_gb300 import moduli32

WORDS = 1 << 25  # words of one operand of the largest call: 2^16 x 32 limbs x 16 polynomials
ELEMENTWISE = {"mulmod": y.YELL_OP_MULMOD, "addmod": y.YELL_OP_ADDMOD, "submod": y.YELL_OP_SUBMOD,
               "muladd": y.YELL_OP_MULADD}
DIRECTIONS = {"forward": y.YELL_FORWARD, "lazy": y.YELL_FORWARD_LAZY, "backward": y.YELL_BACKWARD}


def listed():
    return [
        # one product of the smallest ring in use: launch and call latency
        {"name": "polymul_one", "kind": "polymul", "log_n": 10, "L": 1, "count": 1, "cm0": 0, "gauss": False},
        # a levelled scheme's few limbs, a few products at once
        {"name": "polymul_few", "kind": "polymul", "log_n": 13, "L": 5, "count": 3, "cm0": 0, "gauss": False},
        # the headline batch: 16 products with a noise operand, N = 2^16, 32 limbs
        {"name": "polymul_large", "kind": "polymul", "log_n": 16, "L": 32, "count": 16, "cm0": 0, "gauss": True},
        # a batch of polynomials to the transform domain: 64 x 8 limbs of 2^14
        {"name": "ntt_forward", "kind": "ntt", "log_n": 14, "L": 8, "count": 64, "cm0": 0, "direction": "forward"},
        # a ragged number of small polynomials back, under moduli further down the table
        {"name": "ntt_backward", "kind": "ntt", "log_n": 12, "L": 3, "count": 37, "cm0": 11, "direction": "backward"},
        # one large polynomial kept in lazy form for further additions
        {"name": "ntt_lazy", "kind": "ntt", "log_n": 16, "L": 13, "count": 1, "cm0": 0, "direction": "lazy"},
        # inner products of key switching: accumulate products in the transform domain
        {"name": "muladd", "kind": "elementwise", "log_n": 15, "L": 12, "count": 9, "cm0": 0, "op": "muladd"},
        # requests of all sizes collected into one batch (2^10 .. 2^16, 1 .. 16 limbs)
        {"name": "batch_uneven", "kind": "batch", "count": 512, "lo": 10, "hi": 16, "L": 16, "mix": 4},
        # decryption's last step: coefficients of 16 polynomials as integers below the product of 32 primes
        {"name": "crt_lift", "kind": "crt", "log_n": 16, "L": 32, "count": 16, "cm0": 0},
        # the 32-bit moduli at their largest degree
        {"name": "polymul32", "kind": "polymul32", "log_n": 15, "L": 32, "count": 16, "cm0": 0},
        # RLWE encryptions: samplers, transforms and products of one call sequence
        {"name": "encrypt", "kind": "encrypt", "log_n": 15, "L": 7, "count": 2, "cm0": 0},
        # operands that live in (pinned) host memory: products through the link
        {"name": "polymul_host", "kind": "host", "log_n": 15, "L": 8, "count": 5, "cm0": 0},
    ]


def draw(rng):
    kind = rng.choice(["polymul", "polymul", "ntt", "ntt", "elementwise", "batch", "crt", "polymul32", "encrypt", "host"])
    log = lambda lo, hi: int(round(lo * (hi / lo) ** rng.random()))  # noqa: E731
    if kind == "batch":
        return {"kind": kind, "count": log(16, 512), "lo": 10, "hi": rng.choice([13, 15, 16]), "L": rng.randint(4, 16),
                "mix": rng.randint(1, 1 << 20)}
    lo, hi, most = {"polymul": (10, 17, WORDS), "ntt": (10, 17, WORDS), "elementwise": (10, 16, WORDS),
                    "crt": (10, 16, WORDS), "polymul32": (10, 15, WORDS // 2), "encrypt": (12, 16, WORDS // 8),
                    "host": (12, 16, WORDS // 8)}[kind]
    case = {"kind": kind, "log_n": rng.randint(lo, hi), "L": log(2 if kind == "crt" else 1, 32), "count": log(1, 64),
            "cm0": rng.choice([0, 0, rng.randint(1, 40)])}
    case["count"] = max(1, min(case["count"], most // (case["L"] << case["log_n"])))
    if kind == "polymul":
        case["gauss"] = rng.random() < 0.5
    elif kind == "ntt":
        case["direction"] = rng.choice(list(DIRECTIONS))
    elif kind == "elementwise":
        case["op"] = rng.choice(list(ELEMENTWISE))
    return case


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, count, primes, n, dtype=torch.int64):
    """(count, L, n) words, limb l uniform below primes[l]."""
    t = torch.empty((count, len(primes), n), dtype=dtype, device="cuda")
    for l, p in enumerate(primes):
        t[:, l] = torch.randint(0, int(p), (count, n), generator=g, device="cuda", dtype=torch.int64)
    return t


def _noise(g, count, primes, n):
    """(count, L, n): one integer noise polynomial (sigma 3.2, |e| <= 19) per entry, negatives as p + e."""
    e = (torch.randn((count, 1, n), generator=g, device="cuda") * 3.2).round().clamp(-19, 19).to(torch.int64)
    p = torch.tensor([int(p) for p in primes], dtype=torch.int64, device="cuda").view(1, -1, 1)
    return torch.where(e < 0, p + e, e.expand(-1, len(primes), -1)).contiguous()


def _mix(case):
    r = np.random.RandomState(case["mix"])
    return [(int(r.randint(case["lo"], case["hi"] + 1)), int(r.randint(1, case["L"] + 1))) for _ in range(case["count"])]


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "batch":
        mix = _mix(case)
        for log_n in range(case["lo"], case["hi"] + 1):
            y.init_ntt_tables(log_n, case["L"])
        words = sum(L << log_n for log_n, L in mix)
        a, b, c = (torch.empty(words, dtype=torch.int64, device="cuda") for _ in range(3))
        # residues below the smallest of the moduli are residues of each of them
        least = int(min(y.primes(case["L"])))
        for t in (a, b):
            t.copy_(torch.randint(0, least, (words,), generator=g, device="cuda", dtype=torch.int64))
        items, at = [], 0
        for log_n, L in mix:
            w = L << log_n
            items.append((c[at:at + w], a[at:at + w], b[at:at + w], log_n, L, 0))
            at += w
        return {"kind": kind, "items": items, "c": c}
    log_n, L, count, cm0 = case["log_n"], case["L"], case["count"], case["cm0"]
    n = 1 << log_n
    s = {"kind": kind, "shape": (count, L, log_n, cm0)}
    if kind == "polymul32":
        moduli32.init_ntt_tables(log_n, L, cm0)
        q = moduli32.primes(L, cm0)
        s["a"], s["b"] = (_uniform(g, count, q, n, torch.int32) for _ in range(2))
        s["c"] = torch.empty_like(s["a"])
        return s
    q = y.primes(L, cm0)
    y.init_ntt_tables(log_n, L, cm0)
    if kind == "polymul":
        s["a"] = _uniform(g, count, q, n)
        s["b"] = _noise(g, count, q, n) if case["gauss"] else _uniform(g, count, q, n)
        s["c"] = torch.empty_like(s["a"])
        words = y.polymul_scratch_words(count, L, log_n)
        s["scratch"] = torch.empty(words, dtype=torch.int64, device="cuda") if words else None
    elif kind == "ntt":
        # in place: a further pass takes the words the last one left, which are of the same range
        s["x"], s["direction"] = _uniform(g, count, q, n), DIRECTIONS[case["direction"]]
    elif kind == "elementwise":
        s["op"] = ELEMENTWISE[case["op"]]
        s["a"], s["b"], s["c"] = (_uniform(g, count, q, n) for _ in range(3))
    elif kind == "crt":
        s["x"] = _uniform(g, count, q, n)
        s["out"] = torch.empty((count, n, y.crt_words(L, cm0)), dtype=torch.int64, device="cuda")
    elif kind == "encrypt":
        s["pk"] = tuple(_uniform(g, count, q, n) for _ in range(2))
        s["m"] = torch.randint(0, 1 << 16, (count, 1, n), generator=g, device="cuda").expand(-1, L, -1).contiguous()
        s["u"], s["c0"], s["c1"] = (torch.empty_like(s["m"]) for _ in range(3))
        s["seed"] = seed * 3 + 1
    elif kind == "host":
        for name in ("a", "b", "c"):
            s[name] = torch.empty((count, L, n), dtype=torch.int64, pin_memory=True)
            if name != "c":
                s[name].copy_(_uniform(g, count, q, n))
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        y.dev_polymul_batch(s["items"])
        return s["c"]
    count, L, log_n, cm0 = s["shape"]
    if kind == "polymul":
        y.dev_polymul(s["c"], s["a"], s["b"], count, L, log_n, cm0, scratch=s["scratch"])
        return s["c"]
    if kind == "polymul32":
        moduli32.dev_polymul(s["c"], s["a"], s["b"], count, L, log_n, cm0)
        return s["c"]
    if kind == "ntt":
        y.dev_ntt(s["x"], count, L, log_n, cm0, s["direction"])
        return s["x"]
    if kind == "elementwise":
        y.dev_elementwise(s["op"], s["c"], s["a"], s["b"], count, L, log_n, cm0)
        return s["c"]
    if kind == "crt":
        y.dev_crt_lift(s["out"], s["x"], count, L, log_n, cm0)
        return s["out"]
    if kind == "host":
        a, b, c = (s[k].numpy().view(np.uint64) for k in "abc")
        y.polymul_host(a, b, log_n, cm0, out=c)
        return s["c"]
    # c0 = NTT(e0 + m) + pk0 * NTT(u), c1 = NTT(e1) + pk1 * NTT(u)
    shape = (count, L, log_n, cm0)
    u, c0, c1 = s["u"], s["c0"], s["c1"]
    y.sample_zo(u, *shape, seed=s["seed"])
    y.dev_ntt(u, *shape)
    y.sample_gaussian(c0, *shape, seed=s["seed"] + 1)
    y.dev_elementwise(y.YELL_OP_ADDMOD, c0, c0, s["m"], *shape)
    y.dev_ntt(c0, *shape)
    y.dev_elementwise(y.YELL_OP_MULADD, c0, s["pk"][0], u, *shape)
    y.sample_gaussian(c1, *shape, seed=s["seed"] + 2)
    y.dev_ntt(c1, *shape)
    y.dev_elementwise(y.YELL_OP_MULADD, c1, s["pk"][1], u, *shape)
    return c0, c1


def work(case):
    """Bytes of operands in and results out; operations: the multiplication and two additions of each
    butterfly, and a multiplication (with an addition, for muladd) for each product, on whole residues."""
    kind = case["kind"]
    if kind == "batch":
        mix = _mix(case)
        words = sum(L << log_n for log_n, L in mix)
        return {"bytes": 24 * words, "flops": sum((L << log_n) * (4.5 * log_n + 1) for log_n, L in mix)}
    log_n, L = case["log_n"], case["L"]
    words = case["count"] * L << log_n
    if kind in ("polymul", "host", "polymul32"):
        return {"bytes": (12 if kind == "polymul32" else 24) * words, "flops": words * (4.5 * log_n + 1)}
    if kind == "ntt":
        return {"bytes": 16 * words, "flops": 1.5 * words * log_n}
    if kind == "elementwise":
        return {"bytes": (32 if case["op"] == "muladd" else 24) * words, "flops": 2 * words}
    if kind == "crt":
        return {"bytes": 16 * words, "flops": 2 * words * L}
    # encrypt: the message and both key parts in, both parts of the ciphertext out; three transforms
    return {"bytes": 40 * words, "flops": words * (4.5 * log_n + 5)}


# ---- what run() returns, from integers of any length and without the library ------------------------

def _primes(cm0, L):
    """Primes 2^62 - i 2^21 + 1 in increasing i, from the cm0-th on."""
    def is_prime(m):
        d, r = m - 1, 0
        while d % 2 == 0:
            d, r = d // 2, r + 1
        for b in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
            x = pow(b, d, m)
            if x in (1, m - 1):
                continue
            for _ in range(r - 1):
                x = x * x % m
                if x == m - 1:
                    break
            else:
                return False
        return True

    found, p = [], (1 << 62) + 1
    while len(found) < cm0 + L:
        p -= 1 << 21
        if is_prime(p):
            found.append(p)
    return found[cm0:]


def _negacyclic(a, b, p):
    """a * b mod (X^n + 1, p) by one product of integers with 20 bytes for each coefficient."""
    n, k = len(a), 20
    pack = lambda v: int.from_bytes(b"".join(int(x).to_bytes(k, "little") for x in v), "little")  # noqa: E731
    c = (pack(a) * pack(b)).to_bytes(2 * n * k, "little")
    c = [int.from_bytes(c[i * k:(i + 1) * k], "little") for i in range(2 * n)]
    return [(c[i] - c[i + n]) % p for i in range(n)]


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("polymul", "elementwise", "crt") or (case["count"] * case["L"] << case["log_n"]) > 1 << 17:
        return None  # transforms are pinned by the products; the rest takes too long in this form
    s, count, L = prepare(case, seed), case["count"], case["L"]
    q = _primes(case["cm0"], L)
    host = {k: v.cpu().numpy() for k, v in s.items() if isinstance(v, torch.Tensor) and k in "abcx"}
    if kind == "polymul":
        out = [[_negacyclic(host["a"][i, l], host["b"][i, l], q[l]) for l in range(L)] for i in range(count)]
        return torch.tensor(out, dtype=torch.int64)
    if kind == "elementwise":
        a, b, c = (host[k].astype(object) for k in "abc")
        p = np.array(q, dtype=object).reshape(1, L, 1)
        r = {"mulmod": lambda: a * b, "addmod": lambda: a + b, "submod": lambda: a - b, "muladd": lambda: a * b + c}
        return torch.from_numpy((r[case["op"]]() % p).astype(np.int64))
    Q = 1
    for p in q:
        Q *= p
    lift = [Q // p * pow(Q // p, -1, p) for p in q]
    words = (Q.bit_length() + 63) // 64
    x = host["x"].astype(object)
    total = sum(x[:, l] * lift[l] for l in range(L)) % Q
    raw = b"".join(int(v).to_bytes(8 * words, "little") for v in total.reshape(-1))
    return torch.from_numpy(np.frombuffer(raw, dtype=np.int64).reshape(count, -1, words).copy())
