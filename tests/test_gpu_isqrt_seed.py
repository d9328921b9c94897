"""Square roots of every length around the one-warp root (up to 32 limbs), the
Newton seeds above it (their top 32 limbs), and the steps that one block takes
(up to 448 limbs): perfect squares, their neighbours, values with all bits and
with one bit set."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _limbs(v):
    return np.frombuffer(v.to_bytes(max(1, (v.bit_length() + 31) // 32) * 4, "little"), np.uint32)


@pytest.mark.parametrize("n", list(range(1, 36)) + [45, 46, 61, 62, 63, 64, 65, 66, 67, 90, 129, 200, 333, 439, 441, 446, 447, 448, 449, 450,
                                                        893, 900])
def test_isqrt_of_short_numbers(b2m_gpu, n):
    rng = np.random.default_rng(n)
    r = int.from_bytes(rng.bytes(2 * n), "little") | 1 << (16 * n - 1)
    values = [1 << (32 * n - 32), (1 << (32 * n - 32)) + 1, 1 << (32 * n - 1), (1 << (32 * n)) - 1, r * r - 1, r * r,
              r * r + 1, r * r + 2 * r, (3 << (32 * n - 9)) | 5]
    for v in values:
        got = int.from_bytes(np.asarray(b2m_gpu.isqrt_host(_limbs(v)), np.uint32).tobytes(), "little")
        assert got == math.isqrt(v), hex(v)
