"""Certificates of batches that mix LPs whose arrays are copied from where they
lie (32 KB and more) with small ones, which are gathered on the host: each LP
gets the certificate it gets alone, with points that give x and y, one of them
or neither, in both senses, LPs without rows, columns or entries in between.
The sums of an LP are added in the same order alone and in a batch, except
where its rows cross tiles elsewhere: 1e-12 relative."""
import numpy as np
import pytest

from pramaan_b200.certificate import certify_batch
from pramaan_b200.generators import random_sparse_lp
from pramaan_b200.gnn import WarmStart
from pramaan_b200.pdhg import ModelIR, ObjSense

pytestmark = pytest.mark.gpu

FIELDS = ("objective_value", "primal_residual", "bound_violation", "rel_primal", "rel_dual", "rel_gap",
          "primal_objective", "dual_objective", "kkt")
SMALL, LARGE, TALL = (20, 50, 4), (2500, 6000, 3), (4500, 700, 9)     # 32 KB: 4,096 doubles, 8,192 columns


def _lp(shape, seed):
    if shape is None:
        return ModelIR([1.0, -2.0], [0], [], [], [], [], [0.0, 0.0], [1.0, 1.0], 1, 0.5)
    if shape == "no columns":
        return ModelIR([], [0, 0], [], [], [1.0], [2.0], [], [], 0, 3.0)
    md = random_sparse_lp(*shape, seed=seed)
    md.obj_sense = ObjSense(seed % 2)
    return md


ORDERS = {
    "small": [SMALL] * 40,
    "large_first": [LARGE, SMALL, SMALL, LARGE, TALL, SMALL, None, "no columns"],
    "small_first": [SMALL, None, LARGE, "no columns", SMALL, TALL, LARGE, SMALL],
    "large": [LARGE, TALL, LARGE],
}


@pytest.mark.parametrize("given", ["both", "x", "y", "mixed"])
@pytest.mark.parametrize("order", list(ORDERS))
def test_as_alone(order, given):
    models = [_lp(s, k) for k, s in enumerate(ORDERS[order])]
    rng = np.random.default_rng(1)
    points = []
    for k, md in enumerate(models):
        x = rng.normal(0, 1, md.numVars()) if given in ("both", "x") or (given == "mixed" and k % 3) else None
        y = rng.normal(0, 1, md.numRows()) if given in ("both", "y") or (given == "mixed" and k % 2) else None
        points.append(WarmStart(x, y) if k % 7 != 5 else None)
    got = certify_batch(models, [points, points])
    for k, (md, p) in enumerate(zip(models, points)):
        want = certify_batch([md], [[p]])[0][0]
        for f in FIELDS:
            assert getattr(got[0][k], f) == pytest.approx(getattr(want, f), rel=1e-12, abs=1e-12), (k, f)
            assert getattr(got[0][k], f) == getattr(got[1][k], f)
