"""The warp kernel's giant steps against the oracle: at the edges of a block of
64 passes, on the row-pair product, and on few residue rows over many steps.

With an odd Q every row is active for the primes with (b/p) = -1, so a job of n
sequences at Q = 1 makes exactly n passes a step.  Rows that are residues (some
k*b >= 2^32, fewer than four k) at Q = 2 come in pairs (k, 0), (k, 1) for the
primes with (b/p) = 1, and below T = 128 the second value of a pair is a product
by b.  Up to twelve such rows go through their T/32 steps a lane one by one, in
blocks of up to 32 steps or of several rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(f):
    return [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]


def _check(rs, oracle_mod, base, sign, ks, nmin, width, p0, p1, **opts):
    """The factors of a datless job on [p0, p1], equal to the oracle's; the job's plan and counters."""
    nl = [np.array([nmin, nmin + width - 1], dtype=np.uint32) for _ in ks]
    with rs.Job(base=base, sign=sign, ks=ks, nlists=nl, datless=1, **opts) as job:
        got, st = job.sieve(p0, p1)
        info = dict(job.info)
    want, npr = oracle_mod.Job.from_arrays(base, sign, ks, nl).sieve(p0, p1, datless=True)
    assert st["primes"] == npr
    assert _set(got) == _set(want)
    return info, st, len(want)


@pytest.mark.parametrize("passes", [63, 64, 65, 66, 67, 68, 128, 129])
def test_pass_block_edges(rs, oracle_mod, passes):
    ks = [3 + 2 * i for i in range(passes)]
    info, st, n = _check(rs, oracle_mod, 7, -1, ks, 1000, 20000, 10**6, 10**6 + 20000, Q=1, hash_m=8)
    assert (info["rows"], info["warps_per_prime"]) == (passes, 1) and info["giant_steps"] >= 32
    assert n > 100


@pytest.mark.parametrize("nk,width,T", [(3, 20000, 32), (2, 200000, 128), (1, 70000, 128), (2, 40000, 64)])
def test_row_pair_product(rs, oracle_mod, nk, width, T):
    p0 = 2**33 + 1
    info, st, n = _check(rs, oracle_mod, 745, -1, [9000001 + 2 * i for i in range(nk)], 1000, width, p0, p0 + 3 * 10**7, Q=2)
    assert (info["row_form"], info["warps_per_prime"], info["giant_steps"]) == (0, 1, T)
    assert n >= 3
    assert st["primes"] // 8 < st["paired_primes"] < st["primes"]


@pytest.mark.parametrize("nk,Q,sign,width,hash_m,T", [(1, 2, -1, 60000, 8, 128), (2, 3, 1, 30000, 6, 128),
                                                      (3, 2, -1, 40000, 6, 256), (1, 9, -1, 300000, 7, 256),
                                                      (3, 4, 1, 300000, 7, 512), (1, 3, -1, 200000, 6, 1024),
                                                      (2, 2, -1, 10**6, 6, 4096)])
def test_few_rows_many_steps(rs, oracle_mod, nk, Q, sign, width, hash_m, T):
    ks = [9000001 + 2 * i for i in range(nk)]
    found = 0
    for p0, window in ((10**6, 3 * 10**4), (2**33 + 1, 2 * 10**6), (2**47 + 1, 10**5)):
        info, st, n = _check(rs, oracle_mod, 745, sign, ks, 1000, width, p0, p0 + window, Q=Q, hash_m=hash_m)
        assert (info["row_form"], info["warps_per_prime"], info["giant_steps"]) == (0, 1, T)
        assert info["rows"] <= 12 and st["exact_primes"] <= st["primes"] // 50
        found += n
    assert found > 100


def test_few_rows_batched(rs):
    """The same rows in one batched launch: each item's factors are those of its own run."""
    specs = [(1, 3, 200000, 6), (3, 2, 40000, 6), (1, 9, 300000, 7), (3, 3, 20000, 0)]
    jobs = [rs.Job(base=745, sign=-1, ks=[9000001 + 2 * i for i in range(nk)], datless=1, Q=Q, hash_m=hash_m,
                   nlists=[np.array([1000, 1000 + width - 1], dtype=np.uint32)] * nk, mem_limit=1 << 28)
            for nk, Q, width, hash_m in specs]
    for p0, window in ((10**6, 3 * 10**4), (2**33 + 1, 2 * 10**6)):
        want = [_set(j.sieve(p0, p0 + window)[0]) for j in jobs]
        with rs.Batch() as batch:
            items = [batch.add(j, p0, p0 + window) for j in jobs]
            batch.run()
            assert [_set(batch.result(i)[0]) for i in items] == want and all(map(len, want[:1]))
    for j in jobs:
        j.close()
