"""The cluster kernel that reads its LPs from L2 (halpern_cluster_kernel, the
path of LPs too large for a cluster's shared memory) and the shared-memory one
in the same order of sums.

An LP of 80,640 columns and 27,216 rows fits no cluster's shared memory, and one
such LP in a batch keeps the whole batch off it.  So persistent = 2 runs a set
of small LPs from L2 when the large one is in the batch, and from shared memory
when it is not.  Placed first they lie at the same packed positions both times,
and every LP has its own steps, restarts and sums: the small LPs' iterates have
to be the same bits, rows and columns longer than 16 entries (four lanes of one
kernel, a warp of the other) among them."""
import numpy as np
import pytest

from pramaan_b200 import PdhgOptions, solve_batch
from pramaan_b200.generators import random_sparse_lp, rolling_horizon_lp
from pramaan_b200.pdhg import ALGO_HALPERN
from test_gpu_halpern import _long_rows_and_columns_lp, _with_empty_row
from test_gpu_resident import mixed_lps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def large():
    md = rolling_horizon_lp(336, 80, seed=5)
    # more than 16 blocks of 224 KB at 16 bytes an entry and 20 a row and column
    assert 16 * md.nnz() + 20 * (md.numRows() + md.numVars()) > 16 * (232_448 - 8192)
    return md


def _run(models, persistent, iterations):
    return solve_batch(models, PdhgOptions(persistent=persistent, tolerance=0.0, max_iterations=iterations,
                                           check_frequency=64, algorithm=ALGO_HALPERN))


def test_large_lps_from_l2_follow_the_tiled_path(large):
    """One check interval (no restart yet) against the products over tiles, FP32
    rounding apart, and the same bits from run to run."""
    models = [large, _long_rows_and_columns_lp(), _with_empty_row()]
    a, b, c = _run(models, 2, 64), _run(models, -1, 64), _run(models, 2, 64)
    for p, q, r in zip(a, b, c):
        assert p.iterations == q.iterations == 64
        assert np.allclose(p.x, q.x, rtol=1e-4, atol=1e-4 * (1 + np.abs(q.x).max()))
        assert np.allclose(p.y, q.y, rtol=1e-4, atol=1e-4 * (1 + np.abs(q.y).max()))
        assert np.array_equal(p.x, r.x) and np.array_equal(p.y, r.y)


@pytest.mark.parametrize("iterations", [1, 64, 321])
@pytest.mark.parametrize("which", ["long", "mixed", "rolling"])
def test_both_cluster_kernels_give_the_same_bits(large, which, iterations):
    if which == "long":
        small = [_long_rows_and_columns_lp(seed) for seed in range(2)] + [_with_empty_row()]
    elif which == "mixed":
        small = mixed_lps() + [random_sparse_lp(300, 900, 4, seed=2)]
    else:
        small = [rolling_horizon_lp(T, P, seed=T) for T, P in ((24, 5), (60, 12), (96, 20))]
    shared, l2 = _run(small, 2, iterations), _run(small + [large], 2, iterations)
    for k, (p, q) in enumerate(zip(shared, l2)):
        assert p.iterations == q.iterations and p.restarts == q.restarts, k
        assert np.array_equal(p.x, q.x) and np.array_equal(p.y, q.y), k
