"""Rows by residue and rows as residues, on both sides of the line between them,
against the oracle: the number of k (active rows a residue), the lanes that share
a row, and jobs whose row values would not be staged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,Q,sign,width,T", [(4, 2, -1, 20000, 32), (5, 2, 1, 20000, 32), (3, 4, -1, 20000, 32),
                                               (4, 4, 1, 100000, 32), (5, 4, -1, 100000, 32), (5, 6, -1, 20000, 16),
                                               (9, 6, 1, 20000, 8), (8, 8, -1, 100000, 16), (12, 8, 1, 1000000, 64),
                                               (24, 8, -1, 20000, 4), (24, 7, 1, 20000, 4), (32, 8, -1, 5000, 2),
                                               (48, 5, -1, 5000, 2), (31, 8, 1, 5000, 2)])
def test_line_of_rows_by_residue(rs, oracle_mod, nk, Q, sign, width, T):
    rng = np.random.default_rng(nk * 10 + Q)
    ks = sorted(set((rng.integers(3 * 10**6, 5 * 10**6, 4 * nk) * 2 + 1).tolist()))[:nk]
    nl = [np.array([1000, 1000 + width - 1], dtype=np.uint32) for _ in ks]
    oj = oracle_mod.Job.from_arrays(745, sign, ks, nl)
    found = 0
    with rs.Job(base=745, sign=sign, ks=ks, nlists=nl, datless=1, Q=Q) as job:
        info = job.info
        assert (info["row_form"], info["warps_per_prime"], info["giant_steps"]) == (0, 1, T)
        for p0, window in ((10**6, 2 * 10**4), (2**33 + 1, 10**6), (2**47 + 1, 10**5)):
            got, st = job.sieve(p0, p0 + window)
            want, npr = oj.sieve(p0, p0 + window, datless=True)
            key = lambda f: [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]  # noqa: E731
            assert st["primes"] == npr and key(got) == key(want), p0
            found += len(want)
    assert found > 50
