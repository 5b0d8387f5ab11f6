"""The ordered prime sieve (bits, segment prefix sums, emission) at the edges of
its segments of 2^15 odd numbers, and the sieving primes it builds for large p."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_SEG = 2 * 2**15  # width of one segment


@pytest.mark.parametrize("lo", [3, 10**9 + 7, 2**40 + 1, 2**60 + 12345])
@pytest.mark.parametrize("width", [1, _SEG - 2, _SEG, _SEG + 2, 3 * _SEG, 1100 * _SEG + 6])
def test_segments(rs, oracle_mod, lo, width):
    """Ascending primes over one odd number, a segment less one, exact segments
    and more segments than one scan block takes; too small a buffer reports the
    number needed."""
    if width > 10 * _SEG and lo > 2**41:
        pytest.skip("the oracle takes too long there")
    hi = lo + width - 1
    got = rs.gpu_primes(lo, hi)
    want = oracle_mod.primes(lo, hi)
    assert np.array_equal(got, want)
    if len(want) > 1:
        import ctypes

        n = ctypes.c_size_t(0)
        out = np.zeros(len(want) - 1, dtype=np.uint64)
        rc = rs.lib().rs_gpu_primes(lo, hi, out.ctypes.data, len(out), ctypes.byref(n), 0)
        assert rc == rs.RS_ERR_CAPACITY and n.value == len(want)
