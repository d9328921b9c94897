"""Tables that a call builds do not take the memory that the call itself needs:
what a budget admitted on the 64-bit transforms' smaller or fewer tables it
still admits. Each case in a process of its own, where no table exists yet."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np
import torch
import b200mul
from golden_util import gen_operand

MB = 1000000

def random_limbs(seed, n):
    t = torch.empty(n, dtype=torch.int32, device="cuda")
    b200mul.gen_operand_device(seed, n, 0, t.data_ptr())
    torch.cuda.synchronize()
    return t
"""

# 6,291,456 limbs each: 402.8 MB of workspace. The residue transforms take 201.3
# MB of tables and 9.4 of weights (613.5 in all), the 64-bit ones 201.6 (604.4).
PRODUCT = HEAD + """
b200mul.init(0, 605 * MB)
n = 6 << 20
a, b = random_limbs(1, n), random_limbs(2, n)
def product():
    out = torch.full((2 * n,), -1, dtype=torch.int32, device="cuda")
    b200mul.mul_device(a.data_ptr(), n, b.data_ptr(), n, out.data_ptr(), 2 * n)
    b200mul.stream_check()
    return out
short = product()
b200mul.init(0, 4000 * MB)
assert b200mul.plan_describe(n, n)["launches"] == 6
assert torch.equal(short, product())
print("ok")
"""

# Nodes of 400,000 limbs a value: 136 MB for the merge, of which 35 are taken
# when its first product looks for tables (201.3 MB; the 64-bit ones 50).
MERGE = HEAD + """
b200mul.init(0, 300 * MB)
n = 400000
vals = [[random_limbs(3 * i + f, n) for f in range(3)] for i in range(2)]
def merge():
    nodes = [b200mul.pqt_import([t.data_ptr() for t in v], [n] * 3, 1) for v in vals]
    r = b200mul.pqt_merge(*nodes)
    limbs = [r.limbs(f) for f in range(3)]
    for x in (r, *nodes):
        x.free()
    return limbs
short = merge()
b200mul.init(0, 4000 * MB)
for x, y in zip(short, merge()):
    assert np.array_equal(x, y)
print("ok")
"""


@pytest.mark.parametrize("script", [PRODUCT, MERGE], ids=["product", "merge"])
def test_tables_leave_the_call_its_memory(script):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
