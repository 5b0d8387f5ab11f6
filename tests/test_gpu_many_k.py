"""Jobs of thousands of k, whose primes have hundreds of suspects: their lists
hold them (few primes take the exact path), and the factors are those of the
same k in jobs of a thousand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,width", [(4000, 2000001), (1500, 60000), (5000, 20000)])
def test_many_k(nk, width):
    import rsieve as rs

    rng = np.random.default_rng(nk)
    ks = sorted(set((rng.integers(1, 5 * 10**6, 2 * nk) * 2 + 1).tolist()))[:nk]
    nl = [np.unique(np.concatenate([[10**6, 10**6 + width - 1], rng.integers(10**6, 10**6 + width, 50)])).astype(np.uint32)
          for _ in ks]
    p0 = 2**38 + 1

    def sieve(i, j):
        with rs.Job(base=2, sign=-1, ks=ks[i:j], nlists=nl[i:j], datless=1) as job:
            g, st = job.sieve(p0, p0 + 10**5)
        return {(int(f["p"]), int(f["k"]), int(f["n"])) for f in g}, st

    whole, st = sieve(0, nk)
    parts = set().union(*(sieve(i, min(i + 1000, nk))[0] for i in range(0, nk, 1000)))
    assert st["exact_primes"] <= st["primes"] // 50
    assert whole == parts and (len(whole) > 10 or width < 10**6)
