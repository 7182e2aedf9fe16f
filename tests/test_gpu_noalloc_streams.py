"""Allocation-free products that overlap on two streams.  Products of at most
16,384 entries share nothing, and larger ones without rows of more than 512
entries leave nothing that another call would use: the bits are those of the
calls made one after the other, with operands of very different sizes side by
side (row numbers of one lie beyond the other's rows)."""
import ctypes as C

import numpy as np
import pytest

from pramaan_b200 import _lib as L
from test_zz_no_alloc import csr_from_lengths

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROUNDS = 30


class Product:
    def __init__(self, lens, n, seed):
        rp, ci, v = csr_from_lengths(lens, n, seed)
        self.m, self.n, self.nnz = rp.size - 1, n, int(rp[-1])
        x = np.random.default_rng(seed).standard_normal(n).astype(np.float32)
        self.d = [torch.from_numpy(a).cuda() for a in (rp, ci, v, x)]

    def run(self, stream, y):
        L.check(L.lib().pramaan_spmv_noalloc(*(t.data_ptr() for t in self.d[:3]), self.m, self.n, self.nnz,
                                             self.d[3].data_ptr(), y.data_ptr(), C.c_void_p(stream.cuda_stream)))

    def outputs(self):
        return [torch.full((self.m,), float("nan"), device="cuda") for _ in range(ROUNDS)]


def operands(kind):
    rng = np.random.default_rng(4)
    if kind == "small":      # giant rows on both sides, in the clusters' shared memory
        return [Product(np.concatenate([np.zeros(5000, int), [3000, 0, 2000]]), 900, 1),
                Product(np.array([1500, 2, 0, 700]), 400, 2)]
    if kind == "small_and_large":
        return [Product(np.array([1500, 2, 0, 700]), 400, 2),
                Product(np.concatenate([np.zeros(60_000, int), rng.integers(0, 30, 40_000)]), 5000, 3)]
    return [Product(np.concatenate([np.zeros(60_000, int), rng.integers(0, 30, 40_000)]), 5000, 3),
            Product(rng.integers(0, 500, 900), 7000, 5)]


@pytest.mark.parametrize("kind", ["small", "small_and_large", "large"])
def test_overlapping_calls_keep_their_bits(kind):
    a, b = operands(kind)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    want = []
    for p in (a, b):
        y = p.outputs()[0]
        torch.cuda.synchronize()
        p.run(streams[0], y)
        torch.cuda.synchronize()
        want.append(y)
    got = [a.outputs(), b.outputs()]
    torch.cuda.synchronize()
    for k in range(ROUNDS):
        for p, s, y in zip((a, b), streams, got):
            p.run(s, y[k])
    torch.cuda.synchronize()
    for w, ys in zip(want, got):
        for y in ys:
            assert torch.equal(w.view(torch.int32), y.view(torch.int32))
