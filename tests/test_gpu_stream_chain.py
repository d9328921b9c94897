"""Chains of products through a few device buffers without a host wait in
between, as a caller's own tree runs them: every product reads what the one
before it wrote and overwrites what the one before that read, while kernels of
all three may be resident (csrc/pdl.cuh)."""
import numpy as np
import pytest

from golden_util import gen_operand

pytestmark = pytest.mark.gpu

STEPS = 24


def _int(a):
    return int.from_bytes(np.ascontiguousarray(a, dtype="<u4").tobytes(), "little")


# schoolbook, one block, a cluster, two passes, three passes in five parts
@pytest.mark.parametrize("n", [40, 300, 1500, 5000, 20000, 150000])
def test_each_product_reads_the_one_before_it(b2m_gpu, n):
    torch = pytest.importorskip("torch")
    x, ys = gen_operand(n, n), [gen_operand(n + 1 + i, n) for i in range(4)]
    dev = [torch.from_numpy(y.view(np.int32)).cuda() for y in ys]
    lens = torch.zeros(1, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def chain(wait):
        bufs = [torch.zeros(2 * n, dtype=torch.int32, device="cuda") for _ in range(2)]
        bufs[0][:n] = torch.from_numpy(x.view(np.int32)).cuda()
        torch.cuda.synchronize()
        for i in range(STEPS):
            src, dst = bufs[i % 2], bufs[(i + 1) % 2]
            b2m_gpu.mul_device(src.data_ptr(), n, dev[i % 4].data_ptr(), n, dst.data_ptr(), 2 * n, lens.data_ptr(), s)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return bufs[STEPS % 2].cpu().numpy().view(np.uint32)

    want = chain(True)
    for _ in range(8):
        assert np.array_equal(chain(False), want)
    if n <= 20000:
        v, mask = _int(x), (1 << 32 * n) - 1
        for i in range(STEPS):
            v = (v & mask) * _int(ys[i % 4])
        assert _int(want) == v
