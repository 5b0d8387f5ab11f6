"""A job's chunk buffers over its calls: sized to the first window, grown for
larger ones, and for a window that needs several launches of the first size the
whole window at last; the factors stay the same."""
import pytest

pytestmark = pytest.mark.gpu


def _set(f):
    return {(int(x["p"]), int(x["k"]), int(x["n"])) for x in f}


def test_repeated_window_in_one_launch(rs):
    import rsieve.synth as S

    b, s, ks, nl = S.plain_job(1)
    p0, p1 = 2**33 + 1, 2**33 + 6 * 10**7  # 2.6 million primes, above the 2^21 of a first launch
    with rs.Job(base=b, sign=s, ks=ks, nlists=nl, datless=1) as job:
        calls = [job.sieve(p0, p1) for _ in range(9)]
        assert calls[0][1]["bsgs_launches"] == 2
        assert calls[-1][1]["bsgs_launches"] == 1
        assert all(_set(f) == _set(calls[0][0]) and st["primes"] == calls[0][1]["primes"] for f, st in calls)
        assert len(calls[0][0]) > 100


def test_growing_windows(rs, oracle_mod):
    import rsieve.synth as S

    b, s, ks, nl = S.plain_job(1)
    p0, got, st = 2**33 + 1, None, None
    with rs.Job(base=b, sign=s, ks=ks, nlists=nl, datless=1) as job:
        for width in (10, 10**4, 3 * 10**4, 4 * 10**5, 5 * 10**5, 5 * 10**6):
            got, st = job.sieve(p0, p0 + width - 1)
        again, _ = job.sieve(p0, p0 + 4 * 10**5 - 1)
    oj = oracle_mod.Job.from_arrays(b, s, ks, nl)
    want, npr = oj.sieve(p0, p0 + 5 * 10**6 - 1, datless=True)
    assert st["primes"] == npr and _set(got) == _set(want) and len(want) > 20
    assert _set(again) == {x for x in _set(want) if x[0] < p0 + 4 * 10**5}


@pytest.mark.parametrize("hi", [1000, 20000, 10**5, 3 * 10**6])
def test_window_from_three_in_one_launch(rs, oracle_mod, hi):
    """A window that its buffers hold is one launch, where primes are densest too."""
    import rsieve.synth as S

    b, s, ks, nl = S.plain_job(1)
    with rs.Job(base=b, sign=s, ks=ks[:3], nlists=nl[:3]) as job:
        got, st = job.sieve(3, hi)
    want, npr = oracle_mod.Job.from_arrays(b, s, ks[:3], nl[:3]).sieve(3, hi)
    assert st["bsgs_launches"] == 1 and st["primes"] == npr and _set(got) == _set(want)
