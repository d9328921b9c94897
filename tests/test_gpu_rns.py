"""Products on the three-prime residue transforms (csrc/rns_*.cu), which run
every default plan from 2^14 to 2^27 points of 16-bit digits.

Sizes sit at the edges of the lengths: the shortest and the longest product
of a length, operands longer than half of it (nothing of the first pass is
zero), one-limb operands, squares, and lengths put together from 2, 3, 4, 5,
6 and 8 parts. Up to about a million limbs the oracle gives the product; above
that the 64-bit transform does (the general path, run by fixing one of its
plans). Everything is an integer: results are equal or wrong."""
import numpy as np
import pytest

import oracle
from golden_util import gen_operand

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(a.view(np.int32)).cuda()


def _mul(b2m, torch, a, na, b, nb):
    out = torch.full((na + nb,), -1, dtype=torch.int32, device="cuda")
    olen = torch.zeros(1, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    b2m.mul_device(a.data_ptr(), na, b.data_ptr(), nb, out.data_ptr(), na + nb, olen.data_ptr(), s)
    b2m.stream_check(s)
    return out, int(olen.item())


# 32-bit points 2^13 .. 2^20 (two and three passes), 3 * 2^13, 3 * 2^18, and
# 5 * 2^13, 5 * 2^14, 5 * 2^16, 5 * 2^17 (longest, shortest, unbalanced)
SMALL = [(4096, 1), (8191, 1), (4097, 4095), (8000, 192), (8192, 8192), (16383, 16384), (30000, 2768),
         (65535, 65537), (131072, 131072), (200000, 62144), (262143, 262145), (524288, 524288), (1000000, 48576),
         (12288, 12288), (20000, 4576), (24575, 1), (393216, 393216), (700000, 86432),
         (20480, 20480), (40959, 1), (32000, 769), (40960, 40960), (70000, 11920), (163840, 163840), (300000, 27680),
         (131072, 131073), (327680, 327680)]


@pytest.mark.parametrize("na,nb", SMALL)
@pytest.mark.parametrize("kind", [0, 1])
def test_edges_match_oracle(b2m_gpu, na, nb, kind):
    torch = pytest.importorskip("torch")
    a, b = gen_operand(na + 3, na, kind), gen_operand(nb + 5, nb, kind)
    out, n = _mul(b2m_gpu, torch, _dev(torch, a), na, _dev(torch, b), nb)
    want = oracle.mul_port(a, b)
    got = out.cpu().numpy().view(np.uint32)
    assert n == want.size and np.array_equal(got[:n], want) and not got[n:].any()


@pytest.mark.parametrize("na", [4096, 12288, 70001, 196608, 300000])
def test_squares_match_oracle(b2m_gpu, na):
    torch = pytest.importorskip("torch")
    a = gen_operand(na, na)
    t = _dev(torch, a)
    out, n = _mul(b2m_gpu, torch, t, na, t, na)
    want = oracle.mul_port(a, a)
    assert n == want.size and np.array_equal(out.cpu().numpy().view(np.uint32)[:n], want)


# (sub-)length of the 64-bit transform and one of its non-default plans,
# product sizes; parts of the residue transform in the comment
LARGE = [
    (22, [7, 7, 8], [5, 5, 4], [(1 << 20, 1 << 20), (1900000, 190000)]),             # 2^21: one part
    (23, [7, 8, 8], [5, 4, 4], [(3 << 21, 3 << 21), (12000000, 500000)]),           # 3 * 2^22: 3 weighted parts
    (22, [7, 7, 8], [5, 5, 4], [(3 << 20, 3 << 20), (6000000, 290000)]),             # 3 * 2^21: 3 tree parts
    (22, [7, 7, 8], [5, 5, 4], [(5 << 19, 5 << 19), (5000000, 242880)]),             # 5 * 2^20: 5 tree parts
    (23, [7, 8, 8], [5, 4, 4], [(5 << 20, 5 << 20), (9000000, 1400000)]),            # 5 * 2^21: 5 weighted parts
    (25, [8, 9, 8], [4, 3, 4], [(1 << 23, 1 << 23), (16000000, 700000), (8388609, 8388607)]),  # 2 parts
    (26, [8, 9, 9], [4, 3, 3], [(1 << 24, 1 << 24), (33000000, 500000)]),            # 4 parts
    (25, [8, 9, 8], [4, 3, 4], [(25000000, 25000000), (50000000, 300000)]),          # 3 * 2^24: 6 parts
    (27, [9, 9, 9], [3, 3, 3], [(1 << 25, 1 << 25), (60000000, 7000000)]),           # 8 parts
]


@pytest.mark.parametrize("logn,logr,logc,sizes", LARGE)
@pytest.mark.parametrize("kind", [0, 1])
def test_large_lengths_match_the_64_bit_transform(b2m_gpu, logn, logr, logc, sizes, kind):
    torch = pytest.importorskip("torch")
    for na, nb in sizes:
        a = torch.empty(na, dtype=torch.int32, device="cuda")
        b = torch.empty(nb, dtype=torch.int32, device="cuda")
        b2m_gpu.gen_operand_device(na + 1, na, kind, a.data_ptr())
        b2m_gpu.gen_operand_device(nb + 2, nb, kind, b.data_ptr())
        torch.cuda.synchronize()
        before = b2m_gpu.plan_describe(na, nb)
        assert before["ntt_log2"] == logn and before["logr"] != logr
        out, n = _mul(b2m_gpu, torch, a, na, b, nb)
        try:
            b2m_gpu.set_plan(logn, logr, logc)
            want, nw = _mul(b2m_gpu, torch, a, na, b, nb)
        finally:
            b2m_gpu.set_plan(logn, before["logr"], before["logc"])
        assert n == nw and torch.equal(out, want), (na, nb)


def test_spectrum_sharing_and_batches_use_the_same_path(b2m_gpu):
    """Batched jobs of one length: balanced, unbalanced and one-limb operands
    side by side in one launch."""
    torch = pytest.importorskip("torch")
    sizes = [(8192, 8192), (16000, 300), (16383, 1), (1, 16383), (9000, 7000)]
    ops = [(gen_operand(7 * i + 1, na), gen_operand(7 * i + 2, nb)) for i, (na, nb) in enumerate(sizes)]
    dev = [(_dev(torch, a), _dev(torch, b)) for a, b in ops]
    outs = [torch.full((na + nb,), -1, dtype=torch.int32, device="cuda") for na, nb in sizes]
    jobs = [(a.data_ptr(), na, b.data_ptr(), nb, o.data_ptr(), na + nb, 0)
            for (na, nb), (a, b), o in zip(sizes, dev, outs)]
    b2m_gpu.mul_batch(jobs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for (a, b), o in zip(ops, outs):
        want = oracle.mul_port(a, b)
        assert np.array_equal(o.cpu().numpy().view(np.uint32)[:want.size], want)


@pytest.mark.parametrize("na,nb", [(20480, 20480), (12288, 12288), (90000, 41072), (163840, 163840), (300000, 27680),
                                   (327680, 327680), (393216, 393216), (524288, 524288), (655360, 655360)])
def test_batches_of_one_length_equal_single_products(b2m_gpu, na, nb):
    """Six products of one length in one launch: batched launches are larger,
    and take other tiles than a single product of the length."""
    torch = pytest.importorskip("torch")
    dev, outs, jobs = [], [], []
    for i in range(6):
        a = torch.empty(na, dtype=torch.int32, device="cuda")
        b = torch.empty(nb, dtype=torch.int32, device="cuda")
        b2m_gpu.gen_operand_device(3 * i + 1, na, i % 3 == 2, a.data_ptr())
        b2m_gpu.gen_operand_device(3 * i + 2, nb, 0, b.data_ptr())
        o = torch.full((na + nb,), -1, dtype=torch.int32, device="cuda")
        dev.append((a, b))
        outs.append(o)
        jobs.append((a.data_ptr(), na, b.data_ptr(), nb, o.data_ptr(), na + nb, 0))
    torch.cuda.synchronize()
    b2m_gpu.mul_batch(jobs, torch.cuda.current_stream().cuda_stream)
    for (a, b), o in zip(dev, outs):
        want, _ = _mul(b2m_gpu, torch, a, na, b, nb)
        assert torch.equal(o, want)


def test_served_lengths_belong_to_their_requests(b2m_gpu):
    """Requests of one 3 * 2^k length, some of which 5/6 of it holds, in one
    dispatch: they run in two launches, and every result is its request's."""
    sizes = [(24000, 24000), (20000, 20000), (24576, 20000), (16000, 16900), (20480, 20480), (24576, 24576),
             (33000, 10), (30000, 18000)]
    srv = b2m_gpu.Server(hbm_budget_bytes=2 << 30, streams=1, max_batch=8)
    try:
        for _ in range(3):
            tickets = [srv.submit(na, nb, 100 + i, 200 + i, 0) for i, (na, nb) in enumerate(sizes)]
            for t, (na, nb) in zip(tickets, sizes):
                r = srv.wait(t, 60.0)
                assert r.state == b2m_gpu.DONE and r.residues_ok == 1
                assert na + nb - 1 <= r.out_len <= na + nb, (na, nb, r.out_len)
                srv.release(t)
    finally:
        srv.stop()


# lengths of 2^7 (schoolbook) to 2^12 points: the longest, the shortest,
# unbalanced, and operands longer than half of the length
ONE_LAUNCH = [
    [(1, 1), (64, 64), (1, 127), (127, 1), (33, 2), (3, 5), (100, 28), (31, 32)],
    [(128, 128), (65, 64), (255, 1), (1, 200), (130, 100)],
    [(256, 256), (129, 128), (511, 1), (200, 150), (3, 300)],
    [(512, 512), (257, 256), (1, 1023), (700, 300), (600, 60)],
    [(1024, 1024), (513, 512), (2047, 1), (1500, 400), (90, 1300)],
    [(2048, 2048), (1025, 1024), (1, 4095), (3000, 1000), (4000, 90)],
]


@pytest.mark.parametrize("sizes", ONE_LAUNCH)
@pytest.mark.parametrize("njobs", [1, 63, 64, 255, 511, 514])
def test_batches_of_one_launch_products_match_oracle(b2m_gpu, sizes, njobs):
    """On either side of the counts at which a batch takes another kernel."""
    torch = pytest.importorskip("torch")
    ops = [(gen_operand(5 * i + na, na, kind), gen_operand(7 * i + nb, nb, kind))
           for i, (na, nb) in enumerate(sizes) for kind in (0, 1)]
    dev = [(_dev(torch, a), _dev(torch, b)) for a, b in ops]
    want = [oracle.mul_port(a, b) for a, b in ops]
    jobs, outs = [], []
    lens = torch.full((njobs,), -1, dtype=torch.int64, device="cuda")
    for j in range(njobs):
        a, b = dev[j % len(ops)]
        na, nb = a.numel(), b.numel()
        outs.append(torch.full((na + nb + 1,), -1, dtype=torch.int32, device="cuda"))
        jobs.append((a.data_ptr(), na, b.data_ptr(), nb, outs[j].data_ptr(), na + nb, lens[j:].data_ptr()))
    b2m_gpu.mul_batch(jobs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    lens = lens.cpu().numpy()
    for j, o in enumerate(outs):
        w, got = want[j % len(ops)], o.cpu().numpy().view(np.uint32)
        assert lens[j] == w.size and np.array_equal(got[:w.size], w)
        assert not got[w.size:-1].any() and got[-1] == 0xFFFFFFFF
