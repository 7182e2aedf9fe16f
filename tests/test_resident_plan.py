"""CPU restatement of the shared-memory cluster plan (resident.cu) in NumPy: the
shares of rows and columns, the sub-chunks of 32 elements every block needs, the
entries' positions in its gather vectors and the lines of its short rows.

Checked on random LPs and cluster sizes: shares begin at whole sub-chunks and
cover the LP; every entry's position holds the element its column names once
each owner has stored its sub-chunks into their slots; a block receives exactly
the bytes it waits for; the owner of an element waits for every row that reads it
(what makes overwriting it safe); and the rows a warp sums together begin in
different banks."""
import numpy as np
import pytest

from lp_cases import random_csr

SUB, LONG, NONE = 32, 16, -1


def share_begin(ptr, r0, r1, part, parts):
    if part == 0:
        return r0
    if part == parts:
        return r1
    weight = 2 * (ptr[r0:r1 + 1] - ptr[r0]) + np.arange(r1 - r0 + 1)
    want = int(weight[-1]) * part // parts
    first = int(np.searchsorted(weight[:-1], want))
    return min(r0 + (first + SUB // 2) // SUB * SUB, r1)


def long_stride(n):
    return n + ((2 - n) & 15)


def side(ptr, col, begin, end, base, count):
    """(slots of the sub-chunks a share needs, its entries' positions)."""
    o = col[ptr[begin]:ptr[end]] - base
    need = np.zeros(-(-max(count, 1) // SUB), bool)
    need[o // SUB] = True
    slots = np.where(need, np.cumsum(need) - 1, NONE)
    return slots, slots[o // SUB] * SUB + o % SUB


def transpose(ptr, col, n):
    rows = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))
    order = np.argsort(col, kind="stable")
    return np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))]), rows[order]


CASES = {
    "one_entry": (np.array([1]), 1),
    "short": (np.random.default_rng(0).integers(0, 9, 700), 900),
    "coupling_rows_at_the_end": (np.concatenate([np.full(1500, 3), np.full(60, 48)]), 2000),
    "few_rows": (np.array([40, 0, 17, 16, 3]), 500),
    "no_rows": (np.zeros(0, int), 70),
    "empty_columns": (np.full(100, 2), 4000),
}


@pytest.mark.parametrize("blocks", [1, 2, 3, 6, 16])
@pytest.mark.parametrize("name", list(CASES))
def test_positions_receivers_and_waits(name, blocks):
    lens, n = CASES[name]
    rng = np.random.default_rng(3)
    m = len(lens)
    if m:
        ptr, col, _ = random_csr(m, n, rng, lengths=np.minimum(lens, n))
    else:
        ptr, col = np.zeros(1, np.int64), np.zeros(0, np.int64)
    ptr, col = ptr.astype(np.int64), col.astype(np.int64)
    tptr, trow = transpose(ptr, col, n)
    # an LP inside a batch: rows and columns begin at an offset that is no multiple of 32
    R0, C0 = 37, 91
    P = np.concatenate([np.zeros(R0, np.int64), ptr])
    T = np.concatenate([np.zeros(C0, np.int64), tptr])
    cols, rows = col + C0, trow + R0
    rs = [share_begin(P, R0, R0 + m, b, blocks) for b in range(blocks + 1)]
    cs = [share_begin(T, C0, C0 + n, b, blocks) for b in range(blocks + 1)]
    for s, first, last in ((rs, R0, R0 + m), (cs, C0, C0 + n)):
        assert s[0] == first and s[-1] == last and s == sorted(s)
        assert all((b - first) % SUB == 0 or b == last for b in s)

    xbar, y = rng.integers(1, 10 ** 6, n), rng.integers(1, 10 ** 6, m)
    slot_x, slot_y = {}, {}
    for b in range(blocks):
        slot_x[b], idx = side(P, cols, rs[b], rs[b + 1], C0, n)
        gather = np.zeros((int(slot_x[b].max(initial=NONE)) + 1) * SUB, np.int64)
        received = 0
        for owner in range(blocks):                       # every owner's sub-chunks that this block has a slot for
            for s in range((cs[owner] - C0) // SUB, -(-(cs[owner + 1] - C0) // SUB)):
                if slot_x[b][s] != NONE:
                    own = xbar[s * SUB:(s + 1) * SUB]
                    gather[slot_x[b][s] * SUB:][:len(own)] = own
                    received += SUB * 4
        assert received == 4 * gather.size                # the bytes the block waits for
        assert np.array_equal(gather[idx], xbar[cols[P[rs[b]]:P[rs[b + 1]]] - C0])
        slot_y[b], idx = side(T, rows, cs[b], cs[b + 1], R0, m)
        gather = np.zeros((int(slot_y[b].max(initial=NONE)) + 1) * SUB, np.int64)
        received = 0
        for owner in range(blocks):
            for s in range((rs[owner] - R0) // SUB, -(-(rs[owner + 1] - R0) // SUB)):
                if slot_y[b][s] != NONE:
                    own = y[s * SUB:(s + 1) * SUB]
                    gather[slot_y[b][s] * SUB:][:len(own)] = own
                    received += SUB * 4
        assert received == 4 * gather.size
        assert np.array_equal(gather[idx], y[rows[T[cs[b]]:T[cs[b + 1]]] - R0])

    # the owner of column j has a slot for (so waits for) every row that reads x̄_j, and the other way round
    for i in range(m):
        b = np.searchsorted(rs, R0 + i, side="right") - 1
        for j in col[ptr[i]:ptr[i + 1]]:
            a = np.searchsorted(cs, C0 + j, side="right") - 1
            assert slot_y[a][i // SUB] != NONE and slot_x[b][j // SUB] != NONE


def test_a_column_outside_its_lp_has_no_place():
    """What the batch refuses: the sub-chunk of such a column lies outside the
    LP's table, before it or behind it."""
    ptr, col = np.array([0, 2]), np.array([3, 1200])
    with pytest.raises(IndexError):
        side(ptr, col, 0, 1, 0, 900)
    slots, _ = side(ptr, np.array([3, 200]), 0, 1, 0, 900)
    assert slots[200 // SUB] == 1


@pytest.mark.parametrize("n", range(17, 120))
def test_long_rows_begin_in_different_banks(n):
    step = long_stride(n)
    assert n <= step < n + 16 and step % 16 == 2
    # 8 rows at a time, entries of 8 bytes: 16 pairs of banks
    assert len({(k * step) % 16 for k in range(8)}) == 8
