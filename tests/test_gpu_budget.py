"""Tables that a call builds do not take the memory that the call itself needs:
what a budget admitted beside the 64-bit transforms' tables it still admits.
Where the full residue tables are too large, shorter ones do, and grow later.
Each case in a process of its own, where no table exists yet."""
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

# 6,291,456 limbs each: 402.8 MB of workspace. The residue transforms' full tables
# and weights are 210.7 MB (613.5 in all), the 64-bit ones 201.6 (604.4).
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


# 2^21 points need a table of 25 MB; a graph holds it while a longer product
# replaces it by the full one.
GROWTH = HEAD + """
import oracle
b200mul.init(0, 300 * MB)
n = 524288
a, b = random_limbs(1, n), random_limbs(2, n)
want = oracle.mul_port(*(t.cpu().numpy().view(np.uint32) for t in (a, b)))
out = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
def check():
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32)[:want.size], want)
    out.fill_(-1)
assert b200mul.plan_describe(n, n)["launches"] == 6
bt = b200mul.Batch([(a.data_ptr(), n, b.data_ptr(), n, out.data_ptr(), 2 * n, 0)], b200mul.BATCH_GRAPH)
bt.launch()
check()
assert b200mul.plan_describe(12 * n, 12 * n)["launches"] > 6  # no room for its tables
b200mul.init(0, 4000 * MB)
c = random_limbs(3, 4 * n)
for m in (2 * n, 4 * n):
    big = torch.zeros(2 * m, dtype=torch.int32, device="cuda")
    assert b200mul.plan_describe(m, m)["launches"] == 6
    b200mul.mul_device(c.data_ptr(), m, c.data_ptr(), m, big.data_ptr(), 2 * m)
    b200mul.stream_check()
    p = [int.from_bytes(t.cpu().numpy().tobytes(), "little") for t in (c[:m], big)]
    for q in ((1 << 61) - 1, (1 << 32) - 1, (1 << 32) + 1):
        assert pow(p[0], 2, q) == p[1] % q
    bt.launch()
    check()
    b200mul.mul_device(a.data_ptr(), n, b.data_ptr(), n, out.data_ptr(), 2 * n)
    check()
bt.close()
b200mul.shutdown()
print("ok")
"""


@pytest.mark.parametrize("script", [PRODUCT, MERGE, GROWTH], ids=["product", "merge", "growth"])
def test_tables_leave_the_call_its_memory(script):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
