"""The CTA kernel on residues with rows for few of its warps, against the oracle:
residues side by side (more places than residues, odd numbers of them, of rows), warps
that share a residue's rows or its steps, a single step, one to four rows in
the last pass, and rows whose k have no room beside their ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _key(f):
    return [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]


# (warps a residue, residues side by side, warps for a residue's steps): (1, 4, 4) twice, (1, 8, 2)
# twice, (1, 16, 1) four times, (2, 4, 2), (2, 8, 1), (4, 4, 1) twice, and (1, 16, 1) at the largest Q
@pytest.mark.parametrize("nk,Q,sign,width,T", [(8, 4, 1, 2 * 10**7, 256), (13, 4, -1, 2 * 10**7, 256),
                                               (5, 5, 1, 2 * 10**7, 256), (3, 7, -1, 2 * 10**7, 256),
                                               (2, 9, 1, 2 * 10**7, 256), (5, 15, -1, 2 * 10**7, 256),
                                               (12, 30, 1, 4 * 10**6, 32), (14, 48, -1, 2 * 10**7, 64),
                                               (48, 4, -1, 4 * 10**6, 128), (48, 8, 1, 10**6, 32),
                                               (40, 11, -1, 2 * 10**6, 32), (64, 12, 1, 4 * 10**6, 64),
                                               (1, 3600, -1, 21 * 10**8, 32)])
def test_residues_side_by_side(rs, oracle_mod, nk, Q, sign, width, T):
    rng = np.random.default_rng(nk * 10 + Q)
    ks = sorted(set((rng.integers(3 * 10**6, 5 * 10**6, 4 * nk) * 2 + 1).tolist()))[:nk]
    nl = [np.array([1000, 1000 + width - 1], dtype=np.uint32) for _ in ks]
    oj = oracle_mod.Job.from_arrays(745, sign, ks, nl)
    found = 0
    with rs.Job(base=745, sign=sign, ks=ks, nlists=nl, datless=1, Q=Q) as job:
        info = job.info
        assert (info["warps_per_prime"], info["giant_steps"]) == (16, T)
        for p0, window in ((2**31 + 1, 3 * 10**4), (2**35 + 1, 2 * 10**5), (2**47 + 1, 2 * 10**4)):
            got, st = job.sieve(p0, p0 + window)
            want, npr = oj.sieve(p0, p0 + window, datless=True)
            assert st["primes"] == npr and _key(got) == _key(want), p0
            found += len(want)
    assert found > 20


def test_uneven_residues(rs, oracle_mod):
    """Residues of no row, one and many: row counts far from their mean."""
    rng = np.random.default_rng(5)
    Q, width = 12, 2 * 10**7
    ks = sorted(set((rng.integers(3 * 10**6, 5 * 10**6, 96) * 2 + 1).tolist()))[:24]
    # the k at i has n of the residues i*i and 1 mod Q
    nl = [np.unique(1000 + rng.integers(0, width // Q, 150000) * Q + rng.choice([i * i % Q, 1], 150000)).astype(np.uint32)
          for i in range(24)]
    with rs.Job(base=745, sign=-1, ks=ks, nlists=nl, Q=Q) as job:
        assert (job.info["warps_per_prime"], job.info["rows"]) == (16, sum(1 + (i * i % Q != 1) for i in range(24)))
        got, st = job.sieve(2**28 + 1, 2**28 + 10**6)
    want, npr = oracle_mod.Job.from_arrays(745, -1, ks, nl).sieve(2**28 + 1, 2**28 + 10**6)
    assert st["primes"] == npr and _key(got) == _key(want) and len(want) > 20
