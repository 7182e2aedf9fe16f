"""Empty rows and columns of operands with row-aligned tiles: the tile kernel
does a few per lane, more go to a launch of their own (a thread each).  Both
sides of the rule on A and on A^T, seen in the kernels a profiled iteration
launches; the iterates match the restated reference iteration within the
trajectory tests' 1e-4 * (1 + |ref|)."""
import numpy as np
import pytest

import oracle
from pramaan_b200 import PdhgOptions, Session
from pramaan_b200.pdhg import ModelIR

pytestmark = pytest.mark.gpu

ROWS, COLS, PER = 20_000, 30_000, 3      # about 118 tiles of A: 3 * 32 * 118 = 11,300 empty rows in the tile kernel


def _lp(empty_rows, empty_cols, seed):
    rng = np.random.default_rng(seed)
    m, n = ROWS + empty_rows, COLS + empty_cols
    pr, pc = np.sort(rng.permutation(m)[:ROWS]), np.sort(rng.permutation(n)[:COLS])
    lens = np.zeros(m, np.int64)
    lens[pr] = PER
    ptr = np.concatenate([[0], np.cumsum(lens)])
    # every column is used: a permutation of the columns twice, three entries a row
    col = pc[np.concatenate([rng.permutation(COLS) for _ in range(2)])[:ROWS * PER]]
    val = rng.standard_normal(col.size).astype(np.float32).astype(np.float64)
    # empty rows with y != 0: bounds that 0 violates
    lo, hi = np.full(m, -1e30), np.full(m, 1.0)
    shut = rng.random(m) < 0.3
    lo[shut], hi[shut] = 0.25, 0.5
    return ModelIR(rng.standard_normal(n), ptr, col, val, lo, hi, -rng.random(n), rng.random(n) + 1.0)


@pytest.mark.parametrize("rows, cols", [(0, 0), (9_000, 9_000), (60_000, 500), (500, 60_000), (400_000, 250_000)])
def test_both_sides_of_the_rule(rows, cols):
    md = _lp(rows, cols, rows + cols)
    k = 6
    with Session(md, PdhgOptions(profile_kernels=True)) as s:
        s.iterate(k)
        x, y = s.iterates()
        launches = s.kernel_times()[2]
    assert launches == k * (2 + (rows > 20_000) + (cols > 20_000))
    rx, ry, _ = oracle.trajectory(md, k)
    np.testing.assert_allclose(x, rx, rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(y, ry, rtol=1e-4, atol=1e-4 * (1 + np.abs(ry).max()))
