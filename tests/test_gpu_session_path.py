"""Which path a session's iterations take (Session.path_info), and that LPs on
either side of a limit get the path the rules name: a cluster's shared memory
for LPs whose layout fits it, else products over tiles, row-aligned unless
that takes too many."""
import numpy as np
import pytest

import oracle
from pramaan_b200 import PdhgOptions, Session
from pramaan_b200.generators import random_sparse_lp, zipf_lp
from pramaan_b200.pdhg import ModelIR
from test_gpu_row_tiles import CASES

pytestmark = pytest.mark.gpu


def _path(md, **options):
    with Session(md, PdhgOptions(**options)) as s:
        return s.path_info()


def test_small_lps_run_from_shared_memory():
    for md in (random_sparse_lp(1, 1, 1), random_sparse_lp(200, 600), random_sparse_lp(1000, 3000)):
        assert _path(md)["cluster_blocks"] > 0
        assert _path(md, profile_kernels=True) == {"cluster_blocks": 0, "aligned": (True, True)}


def test_an_lp_that_only_the_estimate_accepts_gets_row_aligned_tiles():
    """120,000 non-zeros: 16 bytes per entry and 36 per row and column fit 16
    blocks, the layout (32-row lines as long as their longest row, gather
    vectors) does not."""
    md = random_sparse_lp(10_000, 30_000, seed=2)
    assert 16 * md.nnz() + 36 * (md.numRows() + md.numVars()) < 16 * (232_448 - 8192)
    with Session(md) as s:
        assert s.path_info() == {"cluster_blocks": 0, "aligned": (True, True)}
        s.iterate(20)
        x, y = s.iterates()
    rx, ry, _ = oracle.trajectory(md, 20)
    np.testing.assert_allclose(x, rx, rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(y, ry, rtol=1e-4, atol=1e-4 * (1 + np.abs(ry).max()))


@pytest.mark.parametrize("name, aligned", [("short", True), ("full_tiles", True), ("long_rows", True), ("cut_tiles", False)])
def test_tiles_hold_whole_rows_unless_they_would_be_too_many(name, aligned):
    lens = CASES[name]
    rng = np.random.default_rng(1)
    m, n = len(lens), 2600
    ptr = np.concatenate([[0], np.cumsum(lens)])
    col = np.concatenate([np.sort(rng.choice(n, size=k, replace=False)) for k in lens])
    md = ModelIR(rng.random(n), ptr, col, rng.standard_normal(len(col)), -np.ones(m), np.ones(m), np.zeros(n), np.ones(n))
    assert _path(md, profile_kernels=True)["aligned"][0] is aligned


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("shape", [(100, 200, 4), (1000, 3000, 4), (5000, 15000, 4)])
def test_calls_of_few_and_of_many_iterations_follow_each_other(shape, graph):
    """Calls of a few iterations run over tiles (loading the LP into a cluster
    would take longer), longer ones on the cluster, on the same iterates."""
    md = random_sparse_lp(*shape, seed=4)
    with Session(md, PdhgOptions(use_graph=graph)) as s:
        assert s.path_info()["cluster_blocks"] > 0
        for k in (1, 1, 9, 2, 5, 1, 20, 3):
            s.iterate(k)
        x, y = s.iterates()
    rx, ry, _ = oracle.trajectory(md, 42)
    np.testing.assert_allclose(x, rx, rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(y, ry, rtol=1e-4, atol=1e-4 * (1 + np.abs(ry).max()))


def test_graph_replay_and_direct_launches_agree_bitwise():
    """The reference iteration over tiles: an LP that no cluster's shared memory
    holds, with rows from one entry to 1,000 (crossing rows), as a CUDA graph and
    launch by launch."""
    md = zipf_lp(20_000, 50_000, cap=1000, seed=8)
    out = []
    for graph in (True, False):
        with Session(md, PdhgOptions(use_graph=graph)) as s:
            assert s.path_info()["cluster_blocks"] == 0
            s.iterate(100)
            out.append(s.iterates())
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_concurrent_captures_match_sequential_ones():
    """Sessions on the tiled products, each capturing its own graph, from four
    threads at once: the bits of the same sessions one after another."""
    from concurrent.futures import ThreadPoolExecutor

    models = [random_sparse_lp(12_000, 36_000, seed=s) for s in range(4)]

    def run(md):
        with Session(md) as s:
            assert s.path_info()["cluster_blocks"] == 0
            for k in (3, 50, 7):     # a capture each
                s.iterate(k)
            return s.iterates()

    one = [run(md) for md in models]
    with ThreadPoolExecutor(4) as ex:
        four = list(ex.map(run, models))
    for a, b in zip(one, four):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
