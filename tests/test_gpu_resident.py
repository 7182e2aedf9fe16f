"""Iterations from a cluster's shared memory (resident.cuh).

The Halpern iteration there keeps the order of the sums of the path it stands
for, so a batch has to give the same bits as with the tiled products
(persistent = -1) after a fixed number of iterations; the LPs cover rows of
every length around the 16 entries of a lane, the 512 of a tile and the length
from which a warp sums a row, empty rows and columns, an LP without rows, and
shares of less than one sub-chunk of 32.  The reference iteration is compared
with the FP64 iteration: after k iterations of FP32 sums and updates, relative
error below k * 2^-20 (an iteration adds a few units of 2^-24 and the method does
not amplify)."""
import numpy as np
import pytest

import oracle
from pramaan_b200 import PdhgOptions, Session, solve_batch
from pramaan_b200.generators import random_sparse_lp, rolling_horizon_batch, rolling_horizon_lp
from pramaan_b200.pdhg import ALGO_HALPERN, ModelIR

pytestmark = pytest.mark.gpu


def lp_of(lengths, n, seed):
    """Feasible LP with the given row lengths (distinct columns, at most n)."""
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(n, size=min(k, n), replace=False)) for k in lengths]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    col = np.concatenate(rows) if len(rows) else np.zeros(0, np.int64)
    val = rng.standard_normal(len(col)).astype(np.float32).astype(np.float64)
    x0 = rng.random(n)
    b = np.array([(val[ptr[i]:ptr[i + 1]] * x0[col[ptr[i]:ptr[i + 1]]]).sum() for i in range(len(rows))])
    ineq = rng.random(len(rows)) < 0.5
    return ModelIR(rng.standard_normal(n), ptr, col, val, np.where(ineq, -1e30, b), b, np.zeros(n), x0 + 1.0)


def mixed_lps():
    rng = np.random.default_rng(5)
    lens = [np.arange(0, 40), rng.integers(0, 70, 300), np.array([1] * 31 + [500, 513, 700, 0, 16, 17, 33]),
            rng.integers(1, 17, 1000), np.array([], np.int64), np.array([3])]
    return [lp_of(k, n, seed) for seed, (k, n) in enumerate(zip(lens, (45, 200, 800, 3000, 7, 2)))]


@pytest.mark.parametrize("iterations", [1, 2, 64, 193])
@pytest.mark.parametrize("which", ["mixed", "rolling", "both"])
def test_halpern_gives_the_bits_of_the_tiled_products(which, iterations):
    models = []
    if which != "rolling":
        models += mixed_lps() * 2
    if which != "mixed":
        models += rolling_horizon_batch(11, seed=3, T_range=(24, 70), P_range=(5, 40))
    o = dict(tolerance=0.0, max_iterations=iterations, check_frequency=64, algorithm=ALGO_HALPERN)
    a = solve_batch(models, PdhgOptions(persistent=0, **o))
    b = solve_batch(models, PdhgOptions(persistent=-1, **o))
    for k, (p, q) in enumerate(zip(a, b)):
        assert p.iterations == q.iterations and p.restarts == q.restarts, k
        assert np.array_equal(p.x, q.x) and np.array_equal(p.y, q.y), k


def test_large_lps_with_constants_in_global_memory():
    """LPs of a cluster each, one of them too large for its constants in shared memory."""
    models = [rolling_horizon_lp(336, 47, seed=1), rolling_horizon_lp(200, 30, seed=2)]
    models += rolling_horizon_batch(8, seed=4, T_range=(24, 40), P_range=(5, 9))
    o = dict(tolerance=0.0, max_iterations=100, check_frequency=64, algorithm=ALGO_HALPERN)
    for p, q in zip(solve_batch(models, PdhgOptions(persistent=0, **o)),
                    solve_batch(models, PdhgOptions(persistent=-1, **o))):
        assert np.array_equal(p.x, q.x) and np.array_equal(p.y, q.y)


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 3, 2), (33, 70, 3), (1000, 3000, 4), (700, 3001, 9), (3000, 9000, 8)])
def test_reference_iteration_against_fp64(shape):
    m, n, per = shape
    md = random_sparse_lp(m, n, min(per, m), seed=m)
    rows = np.repeat(np.arange(m), np.diff(md.row_ptr))
    sums = [np.bincount(i, np.abs(md.values), minlength=k) for i, k in ((rows, m), (md.col_idx, n))]
    sigma, tau = (0.95 / np.where(s > 1e-12, s, 1.0) for s in sums)
    x = np.clip(0.0, md.var_lower, md.var_upper)
    xbar, y = x.copy(), np.zeros(m)
    k = 100
    for _ in range(k):
        w = y / sigma + np.bincount(rows, md.values * xbar[md.col_idx], minlength=m)
        y = sigma * (w - np.clip(w, md.row_lower, md.row_upper))
        new = np.clip(x - tau * (md.obj_coeffs + np.bincount(md.col_idx, md.values * y[rows], minlength=n)),
                      md.var_lower, md.var_upper)
        xbar, x = 2 * new - x, new
    with Session(md, PdhgOptions()) as s:
        s.iterate(k // 2)
        s.iterate(k - k // 2)
        gx, gy = s.iterates()
    for got, want in ((gx, x), (gy, y)):
        assert np.linalg.norm(got - want) <= k * 2.0 ** -20 * max(np.linalg.norm(want), 1e-3)
    ox, oy, _ = oracle.trajectory(md, k)
    assert np.allclose(gx, ox, rtol=1e-4, atol=1e-4)
    assert np.allclose(gy, oy, rtol=1e-4, atol=1e-4 * (1 + abs(oy).max()))


def test_more_clusters_than_fit_at_once_and_the_largest_lps():
    """Several rounds of clusters, an LP that fits only without its constants in
    shared memory, and coupling rows at the end of A (a block of long rows)."""
    rng = np.random.default_rng(8)
    shapes = [(336, 50), (300, 46), (260, 48), (170, 33)] * 2 + [(60, 20), (24, 5)] * 6
    models = [rolling_horizon_lp(T, P, rng=rng) for T, P in shapes]
    o = dict(tolerance=0.0, max_iterations=130, check_frequency=64, algorithm=ALGO_HALPERN)
    a = solve_batch(models, PdhgOptions(persistent=0, **o))
    b = solve_batch(models, PdhgOptions(persistent=-1, **o))
    for p, q in zip(a, b):
        assert p.iterations == q.iterations and p.restarts == q.restarts
        assert np.array_equal(p.x, q.x) and np.array_equal(p.y, q.y)
