"""The allocation-free product on few entries among many empty rows, and on rows
just above the length from which a row is cut at the range boundaries: runs of
empty rows around the strides by which a warp skips them, in front of the
entries, between them and behind, and giant rows of a few pieces and of many
(a lane adds up to 16, a warp more).

Tolerance: a row of L entries is a sum of L rounded products added by some
tree, so |y - exact| <= (L + 1) 2^-24 sum |a x| to first order; twice that is
allowed.  Empty rows are exactly zero."""
import ctypes as C

import numpy as np
import pytest

from pramaan_b200 import _lib as L
from test_zz_no_alloc import csr_from_lengths

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def check(lens, seed):
    n = 20_011
    rp, ci, v = csr_from_lengths(lens, n, seed)
    m, nnz = rp.size - 1, int(rp[-1])
    x = np.random.default_rng(seed + 1).standard_normal(n).astype(np.float32)
    d = [torch.from_numpy(a).cuda() for a in (rp, ci, v, x)]
    y = torch.full((m,), float("nan"), device="cuda")
    L.check(L.lib().pramaan_spmv_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), m, n, nnz, d[3].data_ptr(),
                                         y.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    y = y.cpu().numpy()
    rows = np.repeat(np.arange(m), np.diff(rp))
    terms = v.astype(np.float64) * x[ci]
    want = np.bincount(rows, terms, minlength=m)
    size = np.bincount(rows, np.abs(terms), minlength=m)
    lens = np.diff(rp)
    assert np.all(y[lens == 0] == 0.0)
    assert np.all(np.abs(y - want) <= 2 * (lens + 1) * 2.0 ** -24 * size)


@pytest.mark.parametrize("entries", [1, 300, 20_000])
@pytest.mark.parametrize("run", [31, 32, 33, 64, 1023, 1057, 33_000, 100_001])
def test_runs_of_empty_rows(run, entries):
    rng = np.random.default_rng(run)
    lens = [np.zeros(run, np.int64), rng.integers(1, 4, entries), np.zeros(run + 5, np.int64), rng.integers(0, 3, entries),
            np.zeros(run, np.int64), [2], np.zeros(run, np.int64)]
    check(np.concatenate(lens), run + entries)


def test_one_entry_in_every_thousand_rows():
    check((np.arange(200_000) % 1000 == 7).astype(np.int64), 3)


@pytest.mark.parametrize("length", [513, 600, 1024, 256 * 17, 256 * 18, 256 * 19 + 1, 20_000])
@pytest.mark.parametrize("count", [1, 5, 70])
def test_giant_rows_of_few_and_of_many_pieces(length, count):
    check(np.concatenate([[3, 0], np.tile([length, 0, 2], count), [1]]), length)
