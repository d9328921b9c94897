"""b2m_plan_describe says how many kernels a product launches, before any
product of that length has run as well as after."""
import os
import subprocess
import sys

import pytest

import b200mul

# residue transforms: one launch up to 4,096 limbs, then two kernels a pass
SIZES = [(200, 150, 1), (2048, 2048, 1), (5000, 5000, 4), (60000, 60000, 6), (600000, 600000, 6),
         (3 << 20, 3 << 20, 6), (1 << 24, 1 << 24, 6)]


@pytest.mark.parametrize("na,nb,launches", SIZES)
def test_launches_without_device(na, nb, launches):
    assert b200mul.plan_describe(na, nb)["launches"] == launches


TRACE = """
import sys
import torch
import b200mul
b200mul.init(0)
sizes = %r
first = [b200mul.plan_describe(na, nb)["launches"] for na, nb, _ in sizes]
for (na, nb, want), n in zip(sizes, first):
    a, b, out = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (na, nb, na + nb))
    b200mul.gen_operand_device(1, na, 0, a.data_ptr())
    b200mul.gen_operand_device(2, nb, 0, b.data_ptr())
    ran = len(b200mul.mul_device_traced(a.data_ptr(), na, b.data_ptr(), nb, out.data_ptr(), na + nb))
    assert n == want == ran == b200mul.plan_describe(na, nb)["launches"], (na, nb, n, want, ran)
# the 64-bit transforms of a fixed plan
b200mul.set_plan(16, [7, 9], [5, 3])
assert b200mul.plan_describe(16384, 16384)["launches"] == 6
print("ok")
"""


@pytest.mark.gpu
def test_launches_before_and_after_the_first_product():
    """In a process of its own: the first product of a length builds tables."""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", TRACE % (SIZES,)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
