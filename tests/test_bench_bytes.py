"""bench.py charges each launch the bytes of the transform it belongs to."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

NA, NB, N = 3000, 2000, 1 << 14


# launches of a two-pass product, as b2m_mul_device_traced lists them
RESIDUES = ["fwd_first", "fused_last", "inv_mid", "carry"]
WIDE = ["fwd_first", "fwd_last", "fwd_first", "fused_last", "inv_mid", "carry"]
WIDE3 = ["r3_fwd", "fwd_mid", "fwd_last", "r3_fwd", "fwd_mid", "fused_last", "inv_mid", "inv_mid", "r3_inv", "carry"]


def test_the_transform_is_told_from_its_launches():
    assert bench.is_wide(WIDE) and bench.is_wide(WIDE3)
    assert not bench.is_wide(RESIDUES) and not bench.is_wide(["mul_small"])


def test_residue_launches_add_up_to_the_product():
    got = sum(bench.kernel_bytes(k, NA, NB, N, False) for k in RESIDUES)
    assert got == bench.algorithmic_bytes(NA, NB, N, False) == 8 * (NA + NB) + 48 * N


@pytest.mark.parametrize("kind,want", [("fwd_first", 2 * (NA + NB) + 8 * N), ("r3_fwd", 2 * (NA + NB) + 8 * N),
                                       ("fwd_mid", 16 * N), ("fwd_last", 16 * N), ("inv_mid", 16 * N),
                                       ("r3_inv", 16 * N), ("fused_last", 24 * N), ("carry", 8 * N + 4 * (NA + NB))])
def test_64_bit_launches(kind, want):
    assert bench.kernel_bytes(kind, NA, NB, N, True) == want


def test_64_bit_product():
    assert bench.algorithmic_bytes(NA, NB, N, True) == 8 * (NA + NB) + 64 * N
