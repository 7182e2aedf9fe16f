"""CPU restatement of the row-aligned tiles (align_kernel, CsrDevice::pack_aligned)
in NumPy, with small tiles and segments.

Segments of rows are cut into tiles that hold whole rows where a row fits one
tile; a longer row crosses tiles and is listed with its own row number, its
first tile and its tiles.  The rows are the compacted ones, so the list goes
through the row map, also for an operand whose list of empty rows was trimmed
after the compaction (the panel split keeps only the rows empty in A): what
the tile kernel and the fixup then give every row must be the row's own sum,
once.  Entries are small integers, so the sums are exact."""
import numpy as np
import pytest

TILE = 16
SEGMENT = 4 * TILE


def aligned_tiles(rp_c, row_of):
    """Tiles (first entry, entries, first row, rows ending, continues) and the
    crossing rows (row_of[row], first tile, tiles), as align_kernel makes them."""
    rows_c, nnz = len(rp_c) - 1, int(rp_c[-1])
    tiles, cross = [], []
    segments = -(-nnz // SEGMENT)
    for s in range(segments):
        r = int(np.searchsorted(rp_c, s * SEGMENT))
        r_end = rows_c if s == segments - 1 else int(np.searchsorted(rp_c[:rows_c], (s + 1) * SEGMENT))
        e0 = int(rp_c[r]) if r < r_end else 0
        first = r
        while r < r_end:
            if rp_c[r + 1] - e0 <= TILE:
                r += 1
                continue
            begin, stop = int(rp_c[r]), int(rp_c[r + 1])
            if stop - begin <= TILE:
                tiles.append((e0, begin - e0, first, r - first, 0))
                e0, first = begin, r
                continue
            if begin - e0 == TILE:
                tiles.append((e0, TILE, first, r - first, 0))
                e0, first = begin, r
            at = len(tiles)
            while stop - e0 > TILE:
                tiles.append((e0, TILE, first, r - first, 1))
                e0 += TILE
                first = r
            cross.append((int(row_of[r]), at, len(tiles) - at + 1))
            r += 1
        if first < r_end:
            tiles.append((e0, int(rp_c[r_end]) - e0, first, r_end - first, 0))
    return tiles, cross


def product(rp_c, row_map, empty, entries, tiles, cross):
    """What the tile kernel (whole rows, pieces, empty rows) and the fixup write."""
    out = {}

    def put(row, value):
        assert row not in out, f"row {row} updated twice"
        out[row] = value

    piece = {}   # 2 t: of the row that began earlier, 2 t + 1: of the row that begins in tile t and continues
    for t, (e0, count, first, ending, cont) in enumerate(tiles):
        assert 0 < count <= TILE
        end = e0 + count
        before = rp_c[first] < e0                      # the first row began in an earlier tile
        for i in range(ending):
            b, e = max(int(rp_c[first + i]), e0), int(rp_c[first + i + 1])
            assert e <= end
            total = int(entries[b:e].sum())
            if i == 0 and before:
                piece[2 * t] = total
            else:
                put(int(row_map[first + i]), total)
        if cont:
            begin = int(rp_c[first + ending])
            piece[2 * t + (1 if begin >= e0 else 0)] = int(entries[max(begin, e0):end].sum())
    for r in empty:
        put(int(r), 0)
    for row, at, n in cross:
        put(row, piece[2 * at + 1] + sum(piece[2 * t] for t in range(at + 1, at + n)))
    return out


def lengths(name, rng):
    return {
        "short": rng.integers(0, 6, 300),
        "around_a_tile": np.tile([TILE, 1, TILE - 1, TILE + 1, 0, 3, 2 * TILE, 2 * TILE + 1, 2 * TILE - 1], 4),
        "crossing": np.where(np.arange(200) % 23 == 5, 40, rng.integers(0, 5, 200)),
        "longer_than_a_segment": np.concatenate([rng.integers(0, 5, 50), [3 * SEGMENT, 0, SEGMENT, 90], rng.integers(0, 5, 9)]),
        "only_long": np.full(7, 50),
        "last_is_long": np.concatenate([rng.integers(0, 4, 30), [0, 70]]),
    }[name]


@pytest.mark.parametrize("trimmed", ["all", "some", "none"])
@pytest.mark.parametrize("name", ["short", "around_a_tile", "crossing", "longer_than_a_segment", "only_long", "last_is_long"])
def test_every_row_gets_its_own_sum(name, trimmed):
    rng = np.random.default_rng(len(name))
    lens = lengths(name, rng)
    row_map = np.flatnonzero(lens)
    rp_c = np.concatenate([[0], np.cumsum(lens[row_map])])
    entries = rng.integers(-9, 10, rp_c[-1])
    empty = np.flatnonzero(lens == 0)
    # the panel split drops the rows of its own from the empty ones: they get their value elsewhere
    kept = {"all": empty, "some": empty[::2], "none": empty[:0]}[trimmed]
    tiles, cross = aligned_tiles(rp_c, row_map)
    out = product(rp_c, row_map, kept, entries, tiles, cross)
    ptr = np.concatenate([[0], np.cumsum(lens)])
    assert set(out) == set(row_map.tolist()) | set(kept.tolist())
    for r in out:
        want = int(entries[ptr[r]:ptr[r + 1]].sum())
        assert out[r] == want
    assert sum(t[1] for t in tiles) == rp_c[-1]
    for e0, count, first, ending, cont in tiles:      # a row that fits one tile lies in one tile
        if rp_c[first] < e0:
            assert rp_c[first + 1] - rp_c[first] > TILE


def test_crossing_rows_by_compacted_index_would_be_wrong():
    """Without the map, an operand whose empty rows were all trimmed would list
    a crossing row under its compacted index (rows of 1,500 | 1,200 | 700
    entries, scaled down, the first two of another operand)."""
    lens = np.full(60, 3)
    lens[[10, 20]] = 0
    lens[40] = 40
    row_map = np.flatnonzero(lens)
    rp_c = np.concatenate([[0], np.cumsum(lens[row_map])])
    by_map = aligned_tiles(rp_c, row_map)[1]
    by_index = aligned_tiles(rp_c, np.arange(len(row_map)))[1]
    assert [c[0] for c in by_map] == [40] and [c[0] for c in by_index] == [38]


@pytest.mark.parametrize("entries", [1, 5, 15, 16, 17, 100, 495, 496, 497, 511])
def test_padding_repeats_a_column_of_its_own_load(entries):
    """pad_source: a lane holds 16 consecutive entries and entry j of all lanes is
    one load; padding repeats an entry of the same load, or the last entry where
    the tile has none."""
    for k in range(entries, 512):
        q = k - ((k - entries) // 16 + 1) * 16
        q = q if q >= 0 else entries - 1
        assert 0 <= q < entries
        assert q % 16 == k % 16 or entries < 16
