"""The quadratic-character tables built from squares mod the primes of k'
(square_table_kernel) against characters computed per prime: the same factors.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG = 1760000  # bits of a table segment (kSquareSeg)
SHAPES = {
    # tables of one segment: small, prime powers, squares (all +1), products
    "small": [3, 5, 9, 15, 25, 27, 31, 33, 45, 49, 63, 65, 961, 1155, 3969, 59049, 65535, 262143, 1048573, 1594323],
    # about a segment and several, a prime above a segment with a cofactor, and
    # beyond the largest k' taken (2^25 - 39 is prime, 2^25 + 35 is not taken)
    "segments": [SEG - 1, SEG + 1, SEG - 31, SEG + 31, SEG + 33, 2 * SEG - 1, 2 * SEG + 1, 1759999 * 3, 1760021,
                 3 * 1760021, 9 * 1760021, 5 * 3000017, 7 * 1760021, 4782969, 14348907, 9999991, 9999999, 8999993,
                 2**25 - 39, 2**25 - 1, 2**25 + 35],
}


@pytest.mark.parametrize("base,sign", [(2, -1), (31, 1)])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_tables_from_squares(shape, base, sign):
    import rsieve as rs

    ks = sorted(set(SHAPES[shape]))
    rng = np.random.default_rng(len(shape) + base)
    nl = [np.unique(np.concatenate([[100000, 500000], rng.integers(100000, 500001, 500)])).astype(np.uint32)
          for _ in ks]
    sets = []
    for mode in (rs.TABLES_ALWAYS, rs.TABLES_NEVER):
        with rs.Job(base=base, sign=sign, ks=ks, nlists=nl, datless=1, char_tables=mode) as job:
            g, _ = job.sieve(2**26, 2**26 + 4 * 10**5)
            sets.append({(int(f["p"]), int(f["k"]), int(f["n"])) for f in g})
    assert len(sets[1]) > 500
    assert sets[0] == sets[1]
