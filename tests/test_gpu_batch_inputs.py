"""Malformed LPs inside a batch are refused when they are packed, before the
device sees them: columns outside their own LP (inside the packed batch or not)
and row pointers that do not span the LP's own entries.  The single solve
refuses the same LPs."""
import numpy as np
import pytest

from pramaan_b200 import PdhgOptions, PdhgSolver, solve_batch
from pramaan_b200.generators import random_sparse_lp
from pramaan_b200.pdhg import ALGO_ADAPTIVE, ALGO_HALPERN

pytestmark = pytest.mark.gpu


def _options(algorithm, persistent):
    return PdhgOptions(algorithm=algorithm, persistent=persistent, max_iterations=64, check_frequency=64)


def _bad(kind):
    lp = random_sparse_lp(30, 80, seed=3)
    if kind == "past_the_lp":
        lp.col_idx[5] = 80                    # the next LP's first column
    elif kind == "far_past":
        lp.col_idx[-1] = 160
    elif kind == "negative":
        lp.col_idx[0] = -1                    # the previous LP's last column
    elif kind == "first_pointer":
        lp.row_ptr[0] = 3                     # the previous LP's last row would take three entries
    elif kind == "last_pointer":
        lp.row_ptr[-1] -= 2
    return lp


@pytest.mark.parametrize("algorithm, persistent", [(ALGO_HALPERN, 0), (ALGO_HALPERN, 2), (ALGO_HALPERN, -1), (ALGO_ADAPTIVE, 0)])
@pytest.mark.parametrize("kind", ["past_the_lp", "far_past", "negative", "first_pointer", "last_pointer"])
@pytest.mark.parametrize("place", [0, 1, 2])
def test_refused(kind, place, algorithm, persistent):
    models = [random_sparse_lp(20, 200, seed=k) for k in range(2)]
    models.insert(place, _bad(kind))
    with pytest.raises(ValueError, match="pramaan_lp: (col_idx entry out of bounds|row_ptr must start at 0)"):
        solve_batch(models, _options(algorithm, persistent))
    with pytest.raises(ValueError):
        PdhgSolver(_options(algorithm, persistent)).solve(models[place])


def test_rows_missing_but_entries_given():
    """An LP without rows takes no entries."""
    lp = random_sparse_lp(30, 80, seed=3)
    lp.row_ptr = np.zeros(1, np.int32)
    lp.row_lower = lp.row_upper = np.zeros(0)
    with pytest.raises(ValueError):
        solve_batch([random_sparse_lp(20, 200, seed=1), lp], _options(ALGO_HALPERN, 0))


def test_the_others_still_run():
    """LPs answered without the device (no columns, costs that are not finite)
    keep their answers whatever else they hold."""
    skipped = _bad("past_the_lp")
    skipped.obj_coeffs[0] = np.nan
    out = solve_batch([random_sparse_lp(20, 200, seed=1), skipped], _options(ALGO_HALPERN, 0))
    assert out[0].iterations == 64 and out[1].iterations == 0
