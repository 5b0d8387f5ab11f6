"""The device sieve of a window around the size where its segments change length
(76 segments of 2^16 numbers), with whole and ragged last segments: the number
of primes is the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments", [1, 75, 76, 77, 304, 305])
def test_primes_by_window(rs, oracle_mod, segments):
    import rsieve.synth as S

    b, s, ks, nl = S.plain_job(1)
    with rs.Job(base=b, sign=s, ks=ks[:1], nlists=nl[:1]) as job:
        for p0 in (10**9 + 1, 2**45 + 1):
            for width in (segments * 2**16 - 2, segments * 2**16, segments * 2**16 - 2**14):
                p1 = p0 + width
                assert job.sieve(p0, p1)[1]["primes"] == len(oracle_mod.primes(p0, p1))
