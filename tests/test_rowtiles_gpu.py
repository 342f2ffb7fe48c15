"""lock() of row-grouped inserts through the one-pass tile kernel
(spira_gb300/csrc/spg_rowtiles.cu) at the places where it can go wrong: tiles
filled exactly and overfilled by one, rows longer than a tile, long stretches
of empty rows, buckets that must be split again (clustered columns, many
duplicates) and the widest columns. Bit-exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _columns(kind, rows, n_cols, seed):
    h = gen.hash3(seed, 1, np.arange(len(rows), dtype=np.uint64))
    if kind == "uniform":
        return gen.below(h, n_cols)
    if kind == "equal":  # one column per row
        return (rows.astype(np.uint64) * 7 % n_cols).astype(np.uint32)
    if kind == "few":  # ten columns next to each other
        return (rows.astype(np.uint64) % (n_cols - 10) + h % np.uint64(10)).astype(np.uint32)
    if kind == "band":  # a band around the diagonal
        return ((rows.astype(np.uint64) * 31 + h % np.uint64(400)) % n_cols).astype(np.uint32)
    # geometric clusters: columns 2^k and a few after, so that every split of a
    # bucket leaves one crowded part
    k = (h >> np.uint64(8)) % np.uint64(int(n_cols).bit_length() - 1)
    return np.minimum((np.uint64(1) << k) + h % np.uint64(3), n_cols - 1).astype(np.uint32)


LENGTHS = {
    "edges": [4096, 4095, 1, 1, 4095, 2048, 2048, 2049, 2047, 0, 4097, 31, 32, 33, 0, 12288, 5000, 1, 4064, 32],
    "short": [0, 1, 2, 5, 10, 17, 31, 32, 33] * 700,
    "empty": [3] + [0] * 5000 + [40] + [0] * 2047 + [700] + [0] * 3000,
    "one": [100],
    "long": [2049, 3, 4096, 4097, 2048] * 170,  # more long rows than blocks
}


@pytest.mark.parametrize("kind", ["uniform", "equal", "few", "band", "geometric"])
@pytest.mark.parametrize("lengths", sorted(LENGTHS))
def test_lock_row_tiles(ctx, lengths, kind):
    L = np.asarray(LENGTHS[lengths], np.int64)
    for n_cols in (1000, (1 << 32) - 5):
        rows = np.repeat(np.arange(len(L), dtype=np.uint32), L)
        cols = _columns(kind, rows, n_cols, seed=len(rows))
        vals = gen.sym_unit(gen.hash3(len(rows), 2, np.arange(len(rows), dtype=np.uint64)))
        vals[::11] = 0.0
        vals[5::37] = -0.0
        vals[3::101] = np.nan
        A = sg.Csr(ctx, len(L), n_cols)
        A.lock(rows, cols, vals)
        assert_csr_equal(A.download(), oracle.lock_epochs(len(L), n_cols, [(rows, cols, vals)]))


@pytest.mark.parametrize("order", ["sorted", "grouped"])
@pytest.mark.parametrize("step", [1, 8, 9, 40])
@pytest.mark.parametrize("first,after", [(0, 0), (7, 7), (8, 8), (300, 300)])
def test_lock_offsets_of_spaced_rows(ctx, order, step, first, after):
    """Row offsets written beside the range check up to steps of 8 rows, by a
    pass of their own beyond; empty rows before, between and after."""
    r = first + step * np.arange(700, dtype=np.int64)
    n_rows = int(r[-1]) + 1 + after
    rows = np.repeat(r.astype(np.uint32), 3)
    cols = np.tile(np.array([1, 5, 9] if order == "sorted" else [9, 1, 5], np.uint32), len(r))
    vals = gen.sym_unit(gen.hash3(9, 2, np.arange(len(rows), dtype=np.uint64)))
    for cut in (len(rows), len(rows) - 1, 2):  # whole and ragged 16-byte groups
        A = sg.Csr(ctx, n_rows, 12)
        A.lock(rows[:cut], cols[:cut], vals[:cut])
        assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, 12, [(rows[:cut], cols[:cut], vals[:cut])]))


@pytest.mark.parametrize("order", ["grouped", "shuffled"])
@pytest.mark.parametrize("kind", ["uniform", "band"])
def test_lock_many_short_rows(ctx, kind, order):
    """Above the few-inserts rule: scattered columns by tiles, columns close
    together by the row classes (rows of 0..33 entries)."""
    L = np.tile(np.arange(34, dtype=np.int64), 7500)
    rows = np.repeat(np.arange(len(L), dtype=np.uint32), L)
    n_cols = 9_000_001
    cols = _columns(kind, rows, n_cols, seed=3)
    vals = gen.sym_unit(gen.hash3(4, 2, np.arange(len(rows), dtype=np.uint64)))
    vals[::11] = 0.0
    assert len(rows) > 4 << 20
    if order == "shuffled":
        p = np.argsort(gen.hash3(5, 2, np.arange(len(rows), dtype=np.uint64)), kind="stable")
        rows, cols, vals = rows[p], cols[p], vals[p]
    A = sg.Csr(ctx, len(L), n_cols)
    A.lock(rows, cols, vals)
    assert_csr_equal(A.download(), oracle.lock_epochs(len(L), n_cols, [(rows, cols, vals)]))
