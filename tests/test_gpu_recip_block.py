"""Divisions whose reciprocal ends at, below and above the lengths that one
block takes (33 to 512 limbs of the quotient plus two), by divisors at both
ends of their range: quotient and remainder against Python's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _limbs(v):
    return np.frombuffer(v.to_bytes(max(1, (v.bit_length() + 31) // 32) * 4, "little"), np.uint32)


@pytest.mark.parametrize("m", [27, 29, 30, 31, 32, 60, 61, 62, 63, 64, 65, 125, 126, 127, 128, 200, 253, 254, 255, 333,
                               480, 507, 508, 509, 510, 511, 512, 520])
@pytest.mark.parametrize("n", [5, 40, 700])
def test_quotients_of_m_limbs(b2m_gpu, m, n):
    rng = np.random.default_rng(1000 * m + n)
    top = 1 << (32 * n)
    word = lambda k: int.from_bytes(rng.bytes(4 * k), "little")
    for b in (word(n) | top >> 1, (top >> 1), top - 1, top - (1 << (16 * n)), (word(n) >> 31) | (top >> 32), top // 3):
        for q in (word(m) | 1 << (32 * m - 1), 1 << (32 * m - 32), (1 << (32 * m)) - 1):
            for r in (0, b - 1):
                a = q * b + r
                gq, gr = b2m_gpu.divmod_host(_limbs(a), _limbs(b))
                assert int.from_bytes(np.asarray(gq, np.uint32).tobytes(), "little") == q
                assert int.from_bytes(np.asarray(gr, np.uint32).tobytes(), "little") == r
