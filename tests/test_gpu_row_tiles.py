"""Row-aligned tiles (CsrDevice::pack_aligned) of the reference iteration.

Operands whose rows end at, just before and just after a tile of 512 entries,
rows longer than one tile and longer than a segment of 64 tiles, empty rows and
columns, values with and without an FP32 remainder, and one operand (rows of
300) that would take too many tiles and keeps the cut ones.  profile_kernels
keeps small LPs on the tiled products.  After k iterations of FP32 sums and
updates the relative error against the FP64 iteration stays below k * 2^-20 (an
iteration adds a few units of 2^-24 and the method does not amplify), and the
FP64 residuals of the iterate match the restated ones to 1e-9."""
import numpy as np
import pytest

import oracle
from pramaan_b200 import PdhgOptions, Session
from pramaan_b200.pdhg import ModelIR

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(11)
CASES = {
    "short": RNG.integers(1, 9, 5000),
    "around_a_tile": np.tile([512, 1, 511, 513, 3, 508, 1024, 1025, 1023, 512, 512], 3),
    "full_tiles": np.full(40, 512),
    "long_rows": np.where(np.arange(3000) % 700 == 5, 2500, RNG.integers(0, 6, 3000)),
    "longer_than_a_segment": np.concatenate([RNG.integers(1, 7, 4000), [33000, 0, 40000, 32768], RNG.integers(0, 5, 900)]),
    "cut_tiles": np.full(90, 300),
    "one_entry": np.array([0, 0, 1, 0]),
}


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("name", list(CASES))
def test_reference_iteration_and_residuals(name, exact):
    lens = CASES[name]
    rng = np.random.default_rng(3)
    m, n = len(lens), max(int(lens.max()), 2000) + 37      # 37 or more empty columns
    rows_of = [np.sort(rng.choice(n - 37, size=k, replace=False)) for k in lens]
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate(rows_of).astype(np.int64)
    val = rng.standard_normal(len(col))
    if exact:
        val = val.astype(np.float32).astype(np.float64)
    rows = np.repeat(np.arange(m), lens)
    x0 = rng.random(n)
    b = np.bincount(rows, val * x0[col], minlength=m)
    ineq = rng.random(m) < 0.5
    md = ModelIR(rng.standard_normal(n), ptr, col, val, np.where(ineq, -1e30, b), b, np.zeros(n), x0 + 1.0)

    sums = [np.bincount(i, np.abs(val), minlength=k) for i, k in ((rows, m), (col, n))]
    sigma, tau = (0.95 / np.where(s > 1e-12, s, 1.0) for s in sums)
    x = np.clip(0.0, md.var_lower, md.var_upper)
    xbar, y = x.copy(), np.zeros(m)
    k = 40
    for _ in range(k):
        w = y / sigma + np.bincount(rows, val * xbar[col], minlength=m)
        y = sigma * (w - np.clip(w, md.row_lower, md.row_upper))
        new = np.clip(x - tau * (md.obj_coeffs + np.bincount(col, val * y[rows], minlength=n)), md.var_lower, md.var_upper)
        xbar, x = 2 * new - x, new
    with Session(md, PdhgOptions(profile_kernels=True)) as s:
        s.iterate(k)
        gx, gy = s.iterates()
        pv, dv = s.residuals()
    for got, want in ((gx, x), (gy, y)):
        assert np.linalg.norm(got - want) <= k * 2.0 ** -20 * max(np.linalg.norm(want), 1e-3)
    rpv, rdv = oracle.residuals_ref(md, gx, gy, 1e-6)
    assert pv == pytest.approx(rpv, rel=1e-9, abs=1e-11)
    assert dv == pytest.approx(rdv, rel=1e-9, abs=1e-11)
