"""The baby steps' membership filter and the short baby-step product of the
BSGS kernels, at the sizes where they can go wrong: chains of every remainder,
plans with fewer giant steps than lanes and with several a lane, primes from 3
up, and primes up to 2^63 with factors planted there.

A planted factor: p = k*b^n + sign itself is prime, so p divides the sequence's
term n, which lies inside the job's range."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _is_prime(n):
    if n < 2:
        return False
    small = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)
    for q in small:
        if n % q == 0:
            return n == q
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in small:  # deterministic below 3.3e24
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _set(f):
    return {(int(x["p"]), int(x["k"]), int(x["n"])) for x in f}


def _planted(base, sign, lo, hi, kmax, count, rng):
    """(p, k, n) with p = k*base^n + sign prime in [lo, hi)."""
    got = []
    while len(got) < count:
        p = rng.randrange(lo, hi)
        n = 1
        while p // base**n > kmax:
            n += 1
        k = p // base**n & ~1 | (1 - base % 2)  # p is odd
        q = k * base**n + sign
        if k and lo <= q < hi and _is_prime(q):
            got.append((q, k, n))
    return got


# p ranges around the limits of the products and of the keys (below 2^32 the
# fractions of residues are spaced, above 2^62 only Shoup's product is left)
_P = [(2**31, 2**31 + 2**30), (2**32, 2**32 + 2**31), (2**36, 2**37), (2**43, 2**44), (2**47, 2**48), (2**53, 2**54),
      (2**59, 2**60), (2**61, 2**62), (2**62, 2**62 + 2**61), (2**63 - 2**60, 2**63)]


@pytest.mark.parametrize("base,sign,nk,width", [(2, -1, 3, 40000), (745, -1, 12, 30000), (97, 1, 70, 5000),
                                                (10, -1, 1, 400000), (3, 1, 300, 60000)])
def test_planted_factors(rs, base, sign, nk, width):
    """Every planted factor up to 2^63 is found, and the two baby-step forms
    report the same factors, on warp- and CTA-per-prime plans."""
    rng = random.Random(base)
    plants = [x for lo, hi in _P for x in _planted(base, sign, lo, hi, 10**7, 2, rng)]
    ks = {k for _, k, _ in plants}
    while len(ks) < nk + len(plants):
        ks.add(rng.randrange(3, 10**7) | 1)
    # jobs of nk sequences with a few of the plants each, so that small jobs stay small
    per = max(1, min(nk, 4))
    rest = sorted(ks - {k for _, k, _ in plants})
    for i in range(0, len(plants), per):
        part = plants[i : i + per]
        jk = sorted({k for _, k, _ in part} | set(rest[: max(0, nk - len(part))]))
        nl = [np.arange(1, width, dtype=np.uint32) for _ in jk]
        with rs.Job(base=base, sign=sign, ks=np.array(jk, dtype=np.uint32), nlists=nl) as a, \
                rs.Job(base=base, sign=sign, ks=np.array(jk, dtype=np.uint32), nlists=nl,
                       baby_step=rs.BABY_SHOUP) as b:
            for p, k, n in part:
                lo, hi = max(3, p - 2000), min(p + 2000, 2**63 - 1)
                fa, fb = _set(a.sieve(lo, hi)[0]), _set(b.sieve(lo, hi)[0])
                assert (p, k, n) in fa, (p, k, n, a.info)
                assert fa == fb


@pytest.mark.parametrize("nk,width,hash_m,Q", [(1, 900, 0, 0), (2, 5000, 3, 1), (5, 20000, 8, 2), (3, 60000, 5, 3),
                                               (40, 3000, 7, 2), (9, 70001, 9, 6), (130, 2000, 6, 1)])
def test_filter_shapes(rs, oracle_mod, nk, width, hash_m, Q):
    """Complete factor sets against the oracle from p = 3 up, with baby-step
    counts capped by -m (chains with every remainder, partial last chains) and
    forced Q (giant steps fewer than lanes, several a lane)."""
    import rsieve.synth as S

    b, s, ks, nl = S.make_job(nk * 7 + Q, 31, nk, 3, 5000, 1000, 1000 + width - 1, 0.2)
    oj = oracle_mod.Job.from_arrays(b, s, ks, [np.asarray(x) for x in nl])
    with rs.Job(base=b, sign=s, ks=ks, nlists=nl, hash_m=hash_m, Q=Q) as job:
        for lo, hi in ((3, 3000), (60000, 70000), (10**6, 10**6 + 20000), (2**32 - 20000, 2**32 + 20000)):
            want, npr = oj.sieve(lo, hi)
            got, st = job.sieve(lo, hi)
            assert st["primes"] == npr
            assert _set(got) == _set(want), (lo, job.info)
