"""Jobs of thousands of k against the oracle, on windows with tens of factors:
warp plans whose primes have hundreds of suspects, and a CTA plan whose rows
leave no room in shared memory for the k beside their ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,width,p0,window,cta", [(8000, 2000001, 2**36 + 1, 10**4, True),
                                                    (1500, 60000, 2**33 + 1, 10**5, False),
                                                    (5000, 20000, 2**33 + 1, 10**5, False)])
def test_many_k_oracle(rs, oracle_mod, nk, width, p0, window, cta):
    rng = np.random.default_rng(nk)
    ks = sorted(set((rng.integers(1, 5 * 10**6, 2 * nk) * 2 + 1).tolist()))[:nk]
    nl = [np.array([10**6, 10**6 + width - 1], dtype=np.uint32) for _ in ks]
    with rs.Job(base=2, sign=-1, ks=ks, nlists=nl, datless=1) as job:
        got, st = job.sieve(p0, p0 + window)
        info = dict(job.info)
    # bytes of the rows' ids and k, a baby step's tag and 1.5 words of filter, and
    # the suspects' list (Q is 2): more than a CTA's 227 KB
    need = 6 * info["rows"] + 8 * info["baby_steps"] + 0.016 * info["rows"] / 2 * info["giant_steps"]
    assert info["Q"] == 2 and (info["warps_per_prime"] == 16 and need > 232448) == cta
    want, npr = oracle_mod.Job.from_arrays(2, -1, ks, nl).sieve(p0, p0 + window, datless=True)
    key = lambda f: [(int(x["p"]), int(x["k"]), int(x["n"])) for x in f]  # noqa: E731
    assert st["primes"] == npr and st["exact_primes"] <= npr // 50
    assert key(got) == key(want) and len(want) > 20
