"""The 64-bit transforms where a batch, a tree, a decimal conversion, a division
or the server runs them, and where a product falls back to them.

Default plans run the residue transforms, so the 64-bit kernels with a job
table, the radix-3 step and the spectra that products share are reached under a
plan fixed by b2m_set_plan, and by products whose residue tables do not fit the
budget or are first met by a stream capture. Results are integers and compared
with the oracle, the reference's hashes or Python's own."""
import json
import math
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from golden_util import gen_operand, sha_limbs

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")

# (sub-)length: radices and columns of a plan that is nobody's default
PLANS = {14: ([7, 7], [5, 5]), 15: ([9, 6], [3, 6]), 16: ([7, 9], [5, 3]), 17: ([9, 8], [3, 4]),
         18: ([9, 9], [3, 3]), 19: ([9, 10], [3, 2]), 20: ([10, 10], [2, 2]), 21: ([7, 7, 7], [5, 5, 5])}


@pytest.fixture(scope="module")
def wide(b2m_gpu):
    """Every length from 2^14 to 2^21 points and 3 times those on 64-bit passes."""
    before = {}
    for logn, (logr, logc) in PLANS.items():
        n = 1 << (logn - 2)
        before[logn] = b2m_gpu.plan_describe(n, n)
        b2m_gpu.set_plan(logn, logr, logc)
        assert b2m_gpu.plan_describe(n, n)["launches"] == 3 * len(logr)
        assert b2m_gpu.plan_describe(3 * n, 3 * n)["launches"] == 3 * len(logr) + 3
    yield b2m_gpu
    for logn, d in before.items():
        b2m_gpu.set_plan(logn, d["logr"], d["logc"])


def _int(a):
    return int.from_bytes(np.ascontiguousarray(a, dtype="<u4").tobytes(), "little")


SIZES = [(4096, 4096), (5000, 3000), (8191, 1), (8192, 8192), (16384, 16384), (20000, 9000), (40000, 20000),
         (12288, 12288), (20000, 4000), (24576, 24576), (40000, 9000), (49152, 49152), (90000, 100000),
         (131072, 131072), (393216, 393216), (200, 100)]


@pytest.mark.parametrize("graph", [0, 1])
def test_batches(wide, graph):
    torch = pytest.importorskip("torch")
    ops = [(gen_operand(3 * i + 1, na, i % 3 == 2), gen_operand(3 * i + 2, nb, i % 3 == 2))
           for i, (na, nb) in enumerate(SIZES)]
    dev = [[torch.from_numpy(x.view(np.int32)).cuda() for x in pair] for pair in ops]
    outs = [torch.full((na + nb,), -1, dtype=torch.int32, device="cuda") for na, nb in SIZES]
    lens = torch.full((len(SIZES),), -1, dtype=torch.int64, device="cuda")
    jobs = [(a.data_ptr(), na, b.data_ptr(), nb, o.data_ptr(), na + nb, lens[i:].data_ptr())
            for i, ((na, nb), (a, b), o) in enumerate(zip(SIZES, dev, outs))]
    bt = wide.Batch(jobs, wide.BATCH_GRAPH if graph else 0)
    s = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        for o in outs:
            o.fill_(-1)
        lens.fill_(-1)
        bt.launch(s)
        wide.stream_check(s)
        for i, ((a, b), o) in enumerate(zip(ops, outs)):
            want = oracle.mul_port(a, b)
            got = o.cpu().numpy().view(np.uint32)
            assert int(lens[i]) == want.size and np.array_equal(got[:want.size], want), SIZES[i]
            assert not got[want.size:].any()
    bt.close()


@pytest.mark.parametrize("digits", [100000, 1000000])
def test_tree_levels_with_shared_spectra(wide, digits):
    tr = next(t for t in json.load(open(os.path.join(GOLD, "chudnovsky.json")))["trees"] if t["digits"] == digits)
    r = wide.chudnovsky_bs(0, tr["terms"])
    for which, nm in enumerate("PQT"):
        assert r.lengths[which] == tr[nm]["len"] and sha_limbs(r.limbs(which)) == tr[nm]["sha256"], nm
    r.free()


@pytest.mark.parametrize("na", [9000, 30001])
def test_decimal_levels(wide, na):
    a = gen_operand(na, na)
    limit = sys.get_int_max_str_digits()
    sys.set_int_max_str_digits(0)
    try:
        assert wide.to_decimal_host(a) == str(_int(a))
    finally:
        sys.set_int_max_str_digits(limit)


def test_division_and_root(wide):
    a, b = gen_operand(5, 40000), gen_operand(6, 15001)
    q, r = wide.divmod_host(a, b)
    assert (_int(q), _int(r)) == divmod(_int(a), _int(b))
    assert _int(wide.isqrt_host(a)) == math.isqrt(_int(a))


def test_served_products(wide):
    torch = pytest.importorskip("torch")
    srv = wide.Server(hbm_budget_bytes=2 << 30, streams=2, max_batch=8)
    try:
        todo = []
        for i, (na, nb) in enumerate(SIZES):
            a, b = gen_operand(7 * i + 1, na), gen_operand(7 * i + 2, nb)
            da, db = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
            out = torch.full((na + nb,), -1, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            t = srv.submit(na, nb, a=da.data_ptr(), b=db.data_ptr(), out=out.data_ptr(), out_cap=na + nb)
            todo.append((t, a, b, da, db, out))
        for t, a, b, _, _, out in todo:
            r = srv.wait(t, 60.0)
            want = oracle.mul_port(a, b)
            assert r.state == wide.DONE and r.residues_ok == 1 and r.out_len == want.size
            assert np.array_equal(out.cpu().numpy().view(np.uint32)[:want.size], want)
            srv.release(t)
    finally:
        srv.stop()


# ---- products that fall back: each in a process of its own, where no table of
# the longer lengths exists yet
HEAD = """
import numpy as np
import torch
import b200mul
import oracle
from golden_util import gen_operand

def operands(na, nb, kind):
    a, b = gen_operand(na + 1, na, kind), gen_operand(nb + 2, nb, kind)
    return a, b, *(torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))

def traced(da, db):
    na, nb = da.numel(), db.numel()
    out = torch.full((na + nb,), -1, dtype=torch.int32, device="cuda")
    n = torch.zeros(1, dtype=torch.int64, device="cuda")
    said = b200mul.plan_describe(na, nb)["launches"]
    kinds = [k for k, _, _ in b200mul.mul_device_traced(da.data_ptr(), na, db.data_ptr(), nb, out.data_ptr(), na + nb,
                                                        n.data_ptr())]
    assert said == len(kinds), (said, kinds)
    return out.cpu().numpy().view(np.uint32)[:int(n)], "fwd_last" in kinds
"""

SHORT_BUDGET = HEAD + """
# 2^21 and 3 * 2^20 points: 33 and 50 MB of workspace, 50 and 25 of 64-bit tables;
# the shortest residue tables are 25 and 50 MB, more than a quarter of what is left
for budget, na, nb, kind in ((98, 524288, 524288, 0), (98, 1048575, 1, 0), (195, 600000, 600000, 0),
                             (195, 700000, 500000, 1)):
    b200mul.init(0, budget * 1000000)
    a, b, da, db = operands(na, nb, kind)
    got, wide = traced(da, db)
    assert wide and np.array_equal(got, oracle.mul_port(a, b)), (na, nb)
b200mul.init(0, 300 * 1000000)
assert np.array_equal(b200mul.mul_ntt_cuda(a, b), got)
# shorter ones need no further table
a, b, da, db = operands(60000, 60000, 0)
got, wide = traced(da, db)
assert not wide and np.array_equal(got, oracle.mul_port(a, b))
# a batch under the same budget
sizes = [(524288, 500000), (300000, 300000), (20000, 9000)]
ops = [operands(na, nb, 0) for na, nb in sizes]
outs = [torch.full((na + nb,), -1, dtype=torch.int32, device="cuda") for na, nb in sizes]
b200mul.mul_batch([(x[2].data_ptr(), na, x[3].data_ptr(), nb, o.data_ptr(), na + nb, 0)
                   for (na, nb), x, o in zip(sizes, ops, outs)])
torch.cuda.synchronize()
for x, o in zip(ops, outs):
    want = oracle.mul_port(x[0], x[1])
    assert np.array_equal(o.cpu().numpy().view(np.uint32)[:want.size], want)
print("ok")
"""

CAPTURED_FIRST = HEAD + """
b200mul.init(0)
sizes = [(600000, 600000), (524288, 524000), (5000, 5000), (1500, 1500), (40, 50)]
ops = [operands(na, nb, 0) for na, nb in sizes]
outs = [torch.full((na + nb,), -1, dtype=torch.int32, device="cuda") for na, nb in sizes]
lens = torch.zeros(len(sizes), dtype=torch.int64, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    s = torch.cuda.current_stream().cuda_stream
    for i, ((na, nb), x, o) in enumerate(zip(sizes, ops, outs)):
        b200mul.mul_device(x[2].data_ptr(), na, x[3].data_ptr(), nb, o.data_ptr(), na + nb, lens[i:].data_ptr(), s)
want = [oracle.mul_port(x[0], x[1]) for x in ops]
for _ in range(2):
    for o in outs:
        o.fill_(-1)
    g.replay()
    torch.cuda.synchronize()
    for i, (o, w) in enumerate(zip(outs, want)):
        assert int(lens[i]) == w.size and np.array_equal(o.cpu().numpy().view(np.uint32)[:w.size], w), sizes[i]
got, wide = traced(ops[0][2], ops[0][3])  # outside of the capture the tables are built
assert not wide and np.array_equal(got, want[0])
print("ok")
"""


@pytest.mark.parametrize("script", [SHORT_BUDGET, CAPTURED_FIRST], ids=["short_budget", "captured_first"])
def test_fallback(script):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
