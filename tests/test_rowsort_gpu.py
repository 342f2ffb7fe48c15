"""lock() of inserts in no row order, and of small later epochs
(spira_gb300/csrc/spg_delta.cu): the stable sort by row
(spira_gb300/csrc/spg_rowsort.cu) at its tiles' edges, for one to four digit
passes, with runs of one row, rows too long for the row kernels, and as a later
epoch. Bit-exact against the oracle: the last write of a key depends on the
sort's stability."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _inserts(m, n_rows, n_cols, seed, skew=False):
    ctr = np.arange(m, dtype=np.uint64)
    rows = gen.below(gen.hash3(seed, 1, ctr), n_rows)
    if skew:  # most inserts into one row, in runs
        rows = np.where((ctr // np.uint64(50)) % np.uint64(4) == 0, rows, np.uint32(n_rows // 2)).astype(np.uint32)
    cols = gen.below(gen.hash3(seed, 2, ctr), n_cols)
    vals = gen.sym_unit(gen.hash3(seed, 3, ctr))
    vals[::13] = 0.0
    return rows, cols, vals


@pytest.mark.parametrize("n_rows", [2, 255, 257, 65_537, (1 << 24) + 1])
@pytest.mark.parametrize("m", [3, 1023, 1024, 1025, 70_001])
def test_lock_rows_in_no_order(ctx, n_rows, m):
    first, later = _inserts(m, n_rows, 40, seed=m), _inserts(m, n_rows, 40, seed=m + 1)
    A = sg.Csr(ctx, n_rows, 40)
    A.lock(*first)
    assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, 40, [first]))
    A.lock(*later)
    assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, 40, [first, later]))


@pytest.mark.parametrize("n_rows,n_cols,m,skew", [
    (300_000, 300_000, 2_000_003, False),   # the large tiles, digits of 7 bits
    (300, 400_000, 1_500_003, False),       # of 5
    (4000, 400_000, 1_500_003, False),      # of 6
    (9_000, 500_000, 4_500_000, False),     # more than the few-inserts rule: rows of 500
    (50_000, 1000, 30_000, True),           # one row too long for the row kernels, runs of one row
    (50_000, 100_000, 2_000_003, True),     # of 8
])
def test_lock_rows_in_no_order_large(ctx, n_rows, n_cols, m, skew):
    first, later = _inserts(m, n_rows, n_cols, 5, skew), _inserts(m // 7, n_rows, n_cols, 6, skew)
    A = sg.Csr(ctx, n_rows, n_cols)
    A.lock(*first)
    A.lock(*later)
    assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, n_cols, [first, later]))


@pytest.mark.parametrize("order", ["any", "grouped", "sorted"])
@pytest.mark.parametrize("n_rows,per_row,m", [
    (3000, 50, 1), (3000, 50, 2047), (40, 2500, 2600),   # up to 64 inserts of a row, and more
    (5, 13_000, 300), (4096, 2, 1024), (100_000, 3, 9000), (1, 4096, 64), (1, 4096, 65),
])
def test_lock_small_later_epoch(ctx, n_rows, per_row, m, order):
    """Old entries in whole and ragged chunks of 4096, inserts before the
    first and after the last entry, repeated keys, overwrites and deletes."""
    n_cols = 20_000
    rows = np.repeat(np.arange(n_rows, dtype=np.uint32), per_row)
    ctr = np.arange(len(rows), dtype=np.uint64)
    first = (rows, 1 + gen.below(gen.hash3(1, 1, ctr), n_cols - 2), gen.sym_unit(gen.hash3(1, 2, ctr)))
    r, c, v = _inserts(m, n_rows, n_cols, seed=m)
    k = m // 3  # a third of them on what is there, some twice, some deleted
    at = (gen.hash3(3, 3, np.arange(k, dtype=np.uint64)) % np.uint64(len(rows))).astype(np.int64)
    r[:k], c[:k] = first[0][at], first[1][at]
    v[:k:2] = 0.0
    r[-1], c[-1] = n_rows - 1, n_cols - 1
    r[0], c[0] = 0, 0
    if order != "any":
        o = np.lexsort((c, r)) if order == "sorted" else np.argsort(r, kind="stable")
        r, c, v = r[o], c[o], v[o]
    A = sg.Csr(ctx, n_rows, n_cols)
    A.lock(*first)
    A.lock(r, c, v)
    assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, n_cols, [first, (r, c, v)]))


@pytest.mark.parametrize("n_rows,n_cols,m", [
    (3000, 90, 50_000),            # every column above 32 entries
    (5, 40_000, 60_000),           # source rows of 12 000, columns of one or two
    (20_000, 20_000, 400_000),     # a few columns above 32
    (9000, 1, 9000),               # one column
    (70_000, 300, 2_500_000),      # the large tiles
    (30_000, 4000, 60_000),        # 15 to a column: looked at first
    (30_000, 4000, 64_500),        # above 16: the column sort at once
    (9000, 3_000_000, 9000),       # most columns empty
])
def test_transpose_by_column_sort(ctx, n_rows, n_cols, m):
    first = _inserts(m, n_rows, n_cols, seed=m)
    H = oracle.lock_epochs(n_rows, n_cols, [first])
    A = sg.Csr(ctx, n_rows, n_cols)
    A.load(H.off, H.cols, H.vals)
    assert_csr_equal(A.transpose().download(), oracle.transpose(H))
