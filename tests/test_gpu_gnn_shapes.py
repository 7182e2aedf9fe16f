"""The network's kernels at the edges of what they cut their work into: rows of
32 (a warp's stage), 128 (a dense tile), 256 (a reduction chunk) and one beside,
rows and columns with no, few and many entries, LPs without rows.  Checked
against the NumPy restatement with the tolerances of tests/test_gpu_gnn.py
(relative norms: 1e-2 activations and whole gradient, 3e-2 a block, 1e-3 loss);
sums whose order is part of the definition are compared by their repeatability."""
import numpy as np
import pytest

from oracle import gnn as og
from pramaan_b200.gnn import WarmStartNet
from pramaan_b200.pdhg import ModelIR
from test_gpu_gnn import blocks, check_trace, rel, targets_for

pytestmark = pytest.mark.gpu


def lp(m, n, longest, seed):
    """m x n with row lengths from 0 to `longest` (repeated columns merged)."""
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, n, size=rng.integers(0, longest + 1))) for _ in range(m)]
    if m:
        rows[m // 2] = np.unique(rng.integers(0, n, size=3 * longest))
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    col = np.concatenate(rows) if m else np.zeros(0, np.int64)
    lo = rng.normal(size=m)
    return ModelIR(rng.normal(size=n), ptr, col, rng.normal(size=len(col)), lo, lo + rng.integers(0, 2, m),
                   np.zeros(n), np.full(n, 1e30))


@pytest.mark.parametrize("sizes", [[(1, 1)], [(31, 32), (33, 31)], [(127, 129)], [(128, 128), (0, 5)], [(129, 127)],
                                   [(255, 257), (257, 256)], [(0, 40)], [(700, 90), (5, 1100)]])
def test_forward_and_gradient_at_the_edges(sizes):
    models = [lp(m, n, 9, seed=m + n) for m, n in sizes]
    check_trace(models, seed=3)
    tg = targets_for(models, seed=5)
    net = WarmStartNet(seed=4)
    net.params = og.init_params(4).astype(np.float32)
    graph = net.graph(models, tg)
    loss, grad = net.gradients(graph)
    want_loss, want = og.loss_and_grad(net.params, og.Graph(models, tg), exact=False)
    assert loss == pytest.approx(want_loss, rel=1e-3)
    assert rel(grad, want) < 1e-2
    for name, (b, e) in blocks().items():
        if np.linalg.norm(want[b:e]) > 1e-3 * np.linalg.norm(want):
            assert rel(grad[b:e], want[b:e]) < 3e-2, name
    again_loss, again = net.gradients(graph)
    assert again_loss == loss and np.array_equal(again, grad)
