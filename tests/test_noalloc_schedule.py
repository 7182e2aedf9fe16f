"""CPU restatement of the allocation-free product's schedule (noalloc.cu) in
NumPy: the 32-probe search of a range's rows, the rows a range sums by itself,
the pieces of giant rows (more than two ranges' entries) and the row numbers
the ranges leave for the pass that adds them.

Entries are small integers, so the sums are exact.  Larger products share one
scratch array; the last test lets another call's words appear in it and checks
that a row number is used only where it names a giant row of this call that
begins in that range, so nothing is read or written outside [0, m) and products
without giant rows keep their results."""
import numpy as np
import pytest

TILE = 256


def first_row(rp, m, target):
    """First r in [0, m] with rp[r] >= target, by 32 probes a step; the kernel's
    products are 32 bits wide, the end of a step unsigned."""
    lo, width, steps = 0, m, 0
    while width > 0:
        stride = (width >> 5) + 1
        probes = [rp[lo + q * stride] if q * stride < width else 2 ** 31 - 1 for q in range(32)]
        hit = [q for q in range(32) if probes[q] >= target]
        j = hit[0] if hit else 32
        end = min(j * stride, width)
        begin = (j - 1) * stride + 1 if j > 0 else 0
        assert 31 * stride < 2 ** 31 and j * stride < 2 ** 32 and begin < 2 ** 31
        lo, width, steps = lo + begin, end - begin, steps + 1
    assert steps <= 8
    return lo


def ranges(rp, e, T):
    """(y, words): the rows that ranges write, and per range its piece of an
    earlier giant row, its piece of one that begins here, and that row or -1."""
    m, nnz = len(rp) - 1, int(rp[-1])
    count = -(-nnz // T)
    y, words = {}, np.zeros((count, 3), np.int64)
    for k in range(count):
        last = k == count - 1
        lo, hi = k * T, nnz if last else (k + 1) * T
        r, r1 = first_row(rp, m, lo), m if last else first_row(rp, m, hi)
        assert r == np.searchsorted(rp[:m + 1], lo) or rp[r] >= lo
        words[k, 2] = -1
        if r > 0:
            s, t = rp[r - 1], rp[r]
            if t > lo and t - s > 2 * T:
                words[k, 0] = e[lo:min(t, hi)].sum()
        if r1 > r and rp[r1] - rp[r1 - 1] > 2 * T:
            r1 -= 1
            words[k, 1], words[k, 2] = e[rp[r1]:min(rp[r1 + 1], hi)].sum(), r1
        for i in range(r, r1):
            assert i not in y
            y[i] = int(e[rp[i]:rp[i + 1]].sum())
    return y, words


def finish(rp, T, words, y):
    """finish_giants: adds the pieces of the giant rows."""
    m, nnz = len(rp) - 1, int(rp[-1])
    for k, row in enumerate(words[:, 2]):
        if not 0 <= row < m:
            continue
        s, end = rp[row], min(rp[row + 1], nnz)
        if s < k * T or s >= min((k + 1) * T, nnz) or end - s <= 2 * T:
            continue
        to = min((end - 1) // T, len(words) - 1)
        y[int(row)] = int(words[k, 1] + words[k + 1:to + 1, 0].sum())


def operand(name, rng):
    lens = {
        "short": rng.integers(0, 9, 700),
        "at_the_limit": np.array([2 * TILE, 2 * TILE + 1, 0, 1, TILE, 2 * TILE - 1, 3 * TILE, 5]),
        "giants": np.where(np.arange(400) % 57 == 3, rng.integers(600, 3000, 400), rng.integers(0, 7, 400)),
        "one_giant": np.array([0, 0, 9000, 0]),
        "empty_ends": np.concatenate([np.zeros(700, int), rng.integers(0, 40, 60), np.zeros(900, int)]),
        "giant_last": np.concatenate([rng.integers(0, 5, 90), [1300]]),
    }[name]
    rp = np.concatenate([[0], np.cumsum(lens)])
    return rp, rng.integers(-9, 10, rp[-1])


NAMES = ["short", "at_the_limit", "giants", "one_giant", "empty_ends", "giant_last"]


def sums(rp, e):
    return [int(e[a:b].sum()) for a, b in zip(rp[:-1], rp[1:])]


@pytest.mark.parametrize("tiles", [0.25, 0.5, 1, 3])
@pytest.mark.parametrize("name", NAMES)
def test_every_row_once(name, tiles):
    rp, e = operand(name, np.random.default_rng(5))
    T = int(tiles * TILE)
    y, words = ranges(rp, e, T)
    giants = {int(r) for r in words[:, 2] if r >= 0}
    assert not giants & set(y)
    finish(rp, T, words, y)
    assert [y[i] for i in range(len(rp) - 1)] == sums(rp, e)


@pytest.mark.parametrize("other", NAMES)
@pytest.mark.parametrize("name", NAMES)
def test_another_calls_words_are_not_taken(name, other):
    rng = np.random.default_rng(7)
    rp, e = operand(name, rng)
    rp2, e2 = operand(other, rng)
    rp2 = np.concatenate([np.zeros(10_000, int), rp2])     # row numbers beyond the first call's m
    y, words = ranges(rp, e, TILE)
    foreign = ranges(rp2, e2, TILE)[1]
    want = sums(rp, e)
    giants = {i for i in range(len(rp) - 1) if rp[i + 1] - rp[i] > 2 * TILE}
    for mixed in range(8):
        w, out = words.copy(), dict(y)
        n = min(len(w), len(foreign))
        take = rng.random((n, 3)) < (1.0 if mixed == 0 else 0.5)
        w[:n][take] = foreign[:n][take]
        if mixed == 7:
            w[:, 2] = rng.integers(-2 ** 31, 2 ** 31, len(w))
        finish(rp, TILE, w, out)
        assert set(out) <= set(range(len(rp) - 1))
        assert all(out[i] == want[i] for i in out if i not in giants)


class _Steps:
    """A row_ptr of m + 1 entries that is 0 up to row `at` and 7 from there on."""

    def __init__(self, at):
        self.at = at

    def __getitem__(self, i):
        return 7 if i >= self.at else 0


@pytest.mark.parametrize("m", [2 ** 31 - 1, 2 ** 31 - 2, 2 ** 31 - 32, 2 ** 31 - 33, 2 ** 30 + 1])
def test_search_over_the_most_rows(m):
    """The 32nd stride of a search over 2^31 - 32 rows and more ends at 2^31,
    which is no int."""
    assert 32 * (((2 ** 31 - 32) >> 5) + 1) == 2 ** 31
    for at in (0, 1, 31, 32, m // 2, m - 33, m - 1, m):
        assert first_row(_Steps(at), m, 7) == at
        assert first_row(_Steps(at), m, 0) == 0


def skip_empty(rp, v, r, r1, cleared):
    """skip_empty of the kernel: probes of 32 lanes at growing strides."""
    stride = 32
    while stride <= r1 - r:
        empty = [stride * (q + 1) <= r1 - r and rp[r + stride * (q + 1)] == v for q in range(32)]
        strides = sum(empty)
        assert stride * 32 <= 2 ** 30 and r + stride * strides <= r1
        # the clearing loop's index is unsigned: its last step may pass 2^31
        assert r + stride * strides + 31 < 2 ** 32
        cleared.extend(range(r, r + stride * strides))
        r += stride * strides
        if strides < 32 and stride == 32:
            break
        stride = 32 if strides < 32 else min(stride * 32, 1 << 25)
    return r


@pytest.mark.parametrize("after", [0, 1, 40])
@pytest.mark.parametrize("run", [0, 1, 31, 32, 33, 63, 64, 1023, 1024, 1025, 1056, 1088, 33_000, 33_900, 70_001])
def test_runs_of_empty_rows(run, after):
    """Clears the front of the run and nothing else, and leaves fewer than 32 of
    its rows (or, near the end of the range, fewer than the stride it stood at)."""
    v = 5
    rp = np.concatenate([np.full(run + 1, v), v + 1 + np.arange(after)])
    r1, cleared = len(rp) - 1, []
    r = 0
    for _ in range(8):                       # the kernel comes back after every 32 empty rows
        r = skip_empty(rp, v, r, r1, cleared)
        if r + 32 > r1 or rp[r + 32] != v:
            break
        cleared.extend(range(r, r + 32))
        r += 32
    assert cleared == list(range(r)) and r <= run
    assert run - r < 64


class _Counted(list):
    """Collects ranges without holding them."""

    def __init__(self):
        super().__init__()
        self.rows = 0

    def extend(self, rows):
        self.rows += len(rows)


def test_the_longest_run():
    m = 2 ** 31 - 1
    cleared = _Counted()
    assert skip_empty(_Steps(m), 0, 0, m, cleared) == cleared.rows > m - 2 ** 25
