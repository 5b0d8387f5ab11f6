"""The exact path for primes modulo which the baby step b^Q has an order below,
at and above the number m of baby steps, against the oracle.  A k in the group
that b generates makes every giant step a match, which sends the prime there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _is_prime(n):
    return n > 1 and all(n % q for q in range(2, int(n**0.5) + 1))


def _prime_and_base(d, lo):
    """(p, b): the first prime p = 1 mod d above lo, and an element b > 1 of order d."""
    p = lo // d * d + 1
    while True:
        p += d
        if not _is_prime(p):
            continue
        primes = [q for q in range(2, d + 1) if d % q == 0 and _is_prime(q)]
        for g in range(2, 200):
            b = pow(g, (p - 1) // d, p)
            if b > 1 and all(pow(b, d // q, p) != 1 for q in primes):
                return p, b


@pytest.mark.parametrize("nk,width,hash_m,m", [(8, 60000, 6, 128), (300, 400000, 0, 7168)])
@pytest.mark.parametrize("order", ["2", "3", "31", "m-1", "m", "m+1"])
def test_small_orders(rs, oracle_mod, nk, width, hash_m, m, order):
    d = eval(order, {"m": m})  # noqa: S307
    p, base = _prime_and_base(d, 40000)
    group = sorted({pow(base, e, p) for e in range(min(d, 5))})
    rng = np.random.default_rng(d)
    ks = sorted(set(group) | {int(k) for k in rng.integers(p, 10**6, nk - len(group))})
    nl = [np.unique(np.concatenate([[1000, 1000 + width - 1], rng.integers(1000, 1000 + width, 300)])).astype(np.uint32)
          for _ in ks]
    with rs.Job(base=base, sign=-1, ks=ks, nlists=nl, Q=1, hash_m=hash_m) as job:
        info = job.info
        got, st = job.sieve(p - 50, p + 50)
    assert info["baby_steps"] == m and (info["warps_per_prime"] == 16) == (nk == 300)
    want, npr = oracle_mod.Job.from_arrays(base, -1, ks, nl).sieve(p - 50, p + 50)
    key = lambda f: [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]  # noqa: E731
    assert st["primes"] == npr and st["exact_primes"] > 0
    assert key(got) == key(want) and p in {x[0] for x in key(want)}


def test_smallest_primes(rs, oracle_mod):
    """Primes with more than 64 suspects take the exact path in a job of few probes:
    a prime below m matches at each of its some 170 giant steps."""
    rng = np.random.default_rng(22)
    ks = [1000003 + 2 * i for i in range(22)]
    nl = [np.unique(np.concatenate([[10**6, 10**6 + 70000], rng.integers(10**6, 10**6 + 70001, 3)])).astype(np.uint32)
          for _ in ks]
    with rs.Job(base=745, sign=-1, ks=ks, nlists=nl) as job:
        info = job.info
        got, st = job.sieve(3, 1000)
    assert info["warps_per_prime"] == 1 and info["baby_steps"] > 400 and 300 < info["rows"] * info["giant_steps"] < 600
    want, npr = oracle_mod.Job.from_arrays(745, -1, ks, nl).sieve(3, 1000)
    key = lambda f: [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]  # noqa: E731
    assert st["primes"] == npr and key(got) == key(want) and len(want) > 50
    assert npr // 4 < st["exact_primes"] <= npr
