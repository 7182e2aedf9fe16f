"""Block-diagonal upload from the callers' arrays (csr_upload_f64_parts): every LP of
a mixed batch gets the certificate it gets alone, LPs without rows, columns or
entries between the others; a column outside its LP is refused although it lies
inside the batch, and so are row pointers that decrease."""
import numpy as np
import pytest

from pramaan_b200.certificate import certify_batch
from pramaan_b200.generators import random_sparse_lp
from pramaan_b200.gnn import WarmStart
from pramaan_b200.pdhg import ModelIR

pytestmark = pytest.mark.gpu


def lps():
    free = ModelIR([1.0, -2.0], [0], [], [], [], [], [0.0, 0.0], [1.0, 1.0], 1, 0.5)
    empty = ModelIR([], [0, 0], [], [], [1.0], [2.0], [], [], 0, 3.0)
    zero = ModelIR([1.0, 2.0, 3.0], [0, 0, 0], [], [], [-1.0, 0.5], [1.0, 2.0], [0.0] * 3, [1.0] * 3, 1, 0.0)
    out = [free, empty]
    for m, n, per in ((1, 1, 1), (3, 40, 2), (300, 700, 5)):
        out += [random_sparse_lp(m, n, per, seed=m), zero, empty, free]
    return out


def test_same_certificates_as_alone():
    ms = lps()
    rng = np.random.default_rng(2)
    pts = [WarmStart(rng.normal(0, 1, md.numVars()), rng.normal(0, 1, md.numRows()) if k % 3 else None)
           for k, md in enumerate(ms)]
    for md, p, c in zip(ms, pts, certify_batch(ms, [pts])[0]):
        one = certify_batch([md], [[p]])[0][0]
        for f in ("objective_value", "primal_residual", "bound_violation", "rel_primal", "rel_dual", "rel_gap", "kkt"):
            assert getattr(c, f) == pytest.approx(getattr(one, f), rel=1e-12, abs=1e-13), f


@pytest.mark.parametrize("bad", ["column", "negative", "pointer"])
def test_refused(bad):
    ms = [random_sparse_lp(4, 9, 3, seed=s) for s in range(3)]
    md = ms[0]
    if bad == "pointer":
        md.row_ptr[1] = md.row_ptr[2] + 1
    else:
        md.col_idx[1] = 9 if bad == "column" else -1
    with pytest.raises(Exception, match="col_idx" if bad != "pointer" else "row_ptr"):
        certify_batch(ms, [[None] * 3])
