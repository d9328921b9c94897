"""Decimal conversion at the edges of its quotient correction: values one
below, at and one above powers of ten and multiples of the powers that nodes
are divided by (10^(9 2^j)), where an estimate that is a unit off gives a
remainder outside [0, P), and sizes on either side of one, two and more rounds
of a block and of the grid-wide passes of the top levels. The digits are known
from how the value was made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _limbs(v):
    return np.frombuffer(v.to_bytes((v.bit_length() + 31) // 32 * 4, "little"), np.uint32)


def _check(b2m, v, digits):
    assert b2m.to_decimal_host(_limbs(v)) == digits


@pytest.mark.parametrize("k", [72, 73, 144, 145, 288, 2304, 9 * 2**12, 9 * 2**12 + 1, 100000, 9 * 2**14, 9 * 2**15 - 1,
                               9 * 2**16, 700000, 9 * 2**17 + 5])
def test_powers_of_ten(b2m_gpu, k):
    p = 10**k
    _check(b2m_gpu, p - 1, "9" * k)
    _check(b2m_gpu, p, "1" + "0" * k)
    _check(b2m_gpu, p + 1, "1" + "0" * (k - 1) + "1")


@pytest.mark.parametrize("j", [3, 4, 8, 12, 14, 15, 16])
@pytest.mark.parametrize("d", ["1", "7", "9", "123456789", "499999999"])
def test_multiples_of_node_divisors(b2m_gpu, j, d):
    """q P - 1, q P and q P + 1 with q just below P: the digits of q - 1 and
    then all nines, of q and zeros, of q and a one."""
    k = 9 << j
    q = d + "9" * (k - 1 - len(d)) + "1"
    v = (10 ** (k - 1 - len(d)) * (int(d) + 1) * 10 - 9) * 10**k
    _check(b2m_gpu, v, q + "0" * k)
    _check(b2m_gpu, v + 1, q + "0" * (k - 1) + "1")
    _check(b2m_gpu, v - 1, q[:-1] + "0" + "9" * k)
