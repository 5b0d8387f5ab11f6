"""The prime generator on both sides of the window whose primes come back in one
copy (8192 odd numbers): the oracle's primes, the number needed when the buffer
is too small, and the buffer then left alone."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("odds", [1, 100, 8191, 8192, 8193])
@pytest.mark.parametrize("lo", [3, 10**6 + 1, 10**13 + 1])
def test_small_windows(rs, oracle_mod, lo, odds):
    hi = lo + 2 * (odds - 1)
    want = oracle_mod.primes(lo, hi)
    assert np.array_equal(rs.gpu_primes(lo, hi), want)
    for cap in {0, max(0, len(want) - 1), len(want), len(want) + 7}:
        out, n = np.full(cap + 1, 12345, dtype=np.uint64), ctypes.c_size_t(0)
        rc = rs.lib().rs_gpu_primes(lo, hi, out.ctypes.data if cap else None, cap, ctypes.byref(n), 0)
        assert n.value == len(want) and rc == (rs.RS_OK if cap >= len(want) else rs.RS_ERR_CAPACITY)
        done = len(want) if rc == rs.RS_OK else 0
        assert np.array_equal(out[:done], want[:done]) and (out[done:] == 12345).all()
