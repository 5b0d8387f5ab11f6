"""The CTA kernel when a launch has more tag matches than the list for
settle_kernel holds: a prime left over takes the exact path once, however many
matches it has left.

The base has order three modulo one prime, whose baby steps are three values over and
over, and the 64 giant steps of k = 1 match one in each of the 512 threads'
chains: 32768 tag matches, what the smallest list holds.  The other primes of
the window have some 25 matches each, against room for 11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cube_root_of_one(p):
    return next(x for x in (pow(g, (p - 1) // 3, p) for g in range(2, 100)) if x != 1)


def test_full_candidate_list(rs, oracle_mod):
    p = next(int(q) for q in oracle_mod.primes(4 * 10**6, 4 * 10**6 + 1000) if q % 3 == 1)
    base = _cube_root_of_one(p)
    ks = [1] + [k for k in range(5, 700, 2) if pow(k, 3, p) != 1][:299]
    rng = np.random.default_rng(3)
    nl = [np.unique(np.concatenate([[1000, 400999], rng.integers(1000, 401000, 60)])).astype(np.uint32) for _ in ks]
    with rs.Job(base=base, sign=-1, ks=ks, nlists=nl, Q=1) as job:
        info = job.info
        got, st = job.sieve(p - 400, p + 400)
    assert info["warps_per_prime"] == 16 and info["baby_steps"] >= 3 * 1024 and info["giant_steps"] == 64
    want, npr = oracle_mod.Job.from_arrays(base, -1, ks, nl).sieve(p - 400, p + 400)
    key = lambda f: [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]  # noqa: E731
    assert st["primes"] == npr > 30
    assert key(got) == key(want) and len(want) > 20
    assert 0 < st["exact_primes"] <= st["primes"]
