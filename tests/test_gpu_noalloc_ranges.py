"""The allocation-free product's ranges of rows: sizes around the one-cluster
limit (16,384 entries) and the number of tiles per range, rows around the
giant length (512 entries and up), operands that are not 16-byte aligned,
capture into a CUDA graph.

Tolerance: a row of L entries is a sum of L rounded products added by some
tree, so |y - exact| <= (L + 1) 2^-24 sum |a x| to first order; twice that is
allowed."""
import ctypes as C

import numpy as np
import pytest

from pramaan_b200 import _lib as L
from test_zz_no_alloc import csr_from_lengths

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def lengths_of(kind, nnz, rng):
    """Row lengths that add up to nnz."""
    if kind == "one row":
        return np.array([0, nnz, 0, 0])
    if kind == "giants":      # giant rows next to each other, short and empty rows between some
        out, left = [], nnz
        while left > 0:
            for k in (int(rng.integers(500, 530)), 0, int(rng.integers(1000, 9000)), 3, 1, 0, int(rng.integers(2049, 2200))):
                k = min(k, left)
                out.append(k)
                left -= k
        return np.array(out)
    if kind == "empty runs":
        lens = np.zeros(3 * nnz // 2, np.int64)
        lens[rng.choice(lens.size, nnz // 3, replace=False)] = 3
        lens[-1] += nnz - lens.sum()
        return np.concatenate([lens, np.zeros(100, np.int64)])
    lens = np.minimum(rng.zipf(1.6, size=nnz), 700)
    lens = lens[:np.searchsorted(np.cumsum(lens), nnz)]
    return np.concatenate([lens, [nnz - lens.sum()]])


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("kind", ["one row", "giants", "empty runs", "power law"])
@pytest.mark.parametrize("nnz", [1, 255, 257, 16384, 16385, 100_003, (1 << 21) + 5, (1 << 22) + 1])
def test_every_row_is_summed_once(nnz, kind, offset):
    rng = np.random.default_rng(nnz + offset)
    n = 40_001
    rp, ci, v = csr_from_lengths(lengths_of(kind, nnz, rng), n, seed=nnz)
    m = rp.size - 1
    assert rp[-1] == nnz
    x = rng.standard_normal(n).astype(np.float32)
    dev = torch.device("cuda:0")

    def up(a):   # `offset` elements into its allocation
        buf = torch.zeros(a.size + offset, dtype=torch.from_numpy(a[:1]).dtype, device=dev)
        buf[offset:] = torch.from_numpy(a).to(dev)
        return buf[offset:]

    d = [up(a) for a in (rp, ci, v, x)]
    y = torch.full((m + 2,), 7.0, dtype=torch.float32, device=dev)

    def call(stream):
        L.check(L.lib().pramaan_spmv_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), m, n, nnz,
                                             d[3].data_ptr(), y[1:].data_ptr(), C.c_void_p(stream.cuda_stream)))

    prod = v.astype(np.float64) * x[ci].astype(np.float64)
    rows = np.repeat(np.arange(m), np.diff(rp))
    want = np.bincount(rows, prod, minlength=m)
    room = 2 * (np.diff(rp) + 1) * 2.0 ** -24 * np.bincount(rows, np.abs(prod), minlength=m)
    call(torch.cuda.current_stream())
    first = y.cpu().numpy()
    assert first[0] == 7.0 and first[-1] == 7.0          # nothing outside y is written
    assert np.all(np.abs(first[1:-1] - want) <= room + 1e-37)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        call(stream)
    y.fill_(7.0)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), first)         # fixed order of every sum


def test_a_nan_stays_in_its_rows():
    rng = np.random.default_rng(3)
    rp, ci, v = csr_from_lengths(rng.integers(0, 40, 5000), 3000, seed=3)
    x = rng.standard_normal(3000).astype(np.float32)
    x[17] = np.nan
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(a).to(dev) for a in (rp, ci, v, x)]
    y = torch.empty(5000, dtype=torch.float32, device=dev)
    L.check(L.lib().pramaan_spmv_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), 5000, 3000, len(v),
                                         d[3].data_ptr(), y.data_ptr(), None))
    torch.cuda.synchronize()
    has = np.bincount(np.repeat(np.arange(5000), np.diff(rp)), ci == 17, minlength=5000) > 0
    assert np.array_equal(np.isnan(y.cpu().numpy()), has)
