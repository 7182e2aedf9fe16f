"""Column-panel splits whose short part holds rows longer than a tile (512
entries): with panel_split = 1,000, rows of 513 to 999 entries cross the tiles
of the short rows' operand.  The long rows are empty in that operand without
being empty in A, so the crossing rows' numbers go through its row map; LPs
with and without rows that are empty in A.  Iterates match the restated
reference iteration within 1e-4 * (1 + |ref|), the panel tests' tolerance."""
import numpy as np
import pytest

from lp_cases import random_csr
from test_gpu_panel import _check_oracle, _feasible, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("empty", [0, 40])
@pytest.mark.parametrize("split", [513, 1000])
def test_crossing_rows_of_the_short_part(split, empty):
    m, n = 4000, 50_000
    rng = np.random.default_rng(split + empty)
    lens = rng.integers(1, 7, m)
    at = rng.choice(m, 60, replace=False)
    lens[at[:20]] = rng.integers(1000, 3000, 20)     # long rows at either threshold
    lens[at[20:]] = rng.integers(513, 1000, 40)      # short rows at 1,000
    lens[rng.choice(np.setdiff1d(np.arange(m), at), empty, replace=False)] = 0
    rp, ci, v = random_csr(m, n, rng, lengths=lens)
    model = _feasible(rp, ci, v, m, n, 7)
    info, x, y = _run(model, 12, split)
    assert info["panels"] > 0 and info["min_len"] == split
    assert info["long_rows"] == int((lens >= split).sum())
    _check_oracle(model, 12, x, y, f"rows of {split} and more long, {empty} empty rows")
