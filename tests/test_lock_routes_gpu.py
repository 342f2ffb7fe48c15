"""lock()'s choice between its ways for row-grouped inserts, at the edges of
each rule. Bit-exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def test_lock_many_clustered_rows_of_wide_columns(ctx):
    """More inserts than the few-inserts rule, columns close together but
    wider than the row classes take: by tiles, in any order and grouped."""
    n, n_cols = 1_100_000, (1 << 27) + 3
    rows = np.repeat(np.arange(n, dtype=np.uint32), 4)
    ctr = np.arange(len(rows), dtype=np.uint64)
    cols = (rows.astype(np.uint64) * np.uint64(120) + gen.hash3(7, 1, ctr) % np.uint64(6)).astype(np.uint32)
    vals = gen.sym_unit(gen.hash3(7, 2, ctr))
    vals[::11] = 0.0
    assert len(rows) > 4 << 20
    p = np.argsort(gen.hash3(7, 3, ctr), kind="stable")
    for e in ((rows, cols, vals), (rows[p], cols[p], vals[p])):
        A = sg.Csr(ctx, n, n_cols)
        A.lock(*e)
        assert_csr_equal(A.download(), oracle.lock_epochs(n, n_cols, [e]))


def _hub_inserts(n_rows, n_cols, hubs, seed, per_row=3):
    """per_row inserts into every row and, at `hubs`' rows, so many more."""
    L = np.full(n_rows, per_row, np.int64)
    for r, k in hubs:
        L[r] += k
    rows = np.repeat(np.arange(n_rows, dtype=np.uint32), L)
    ctr = np.arange(len(rows), dtype=np.uint64)
    vals = gen.sym_unit(gen.hash3(seed, 2, ctr))
    vals[::7] = 0.0
    vals[::101] = np.nan
    return rows, gen.below(gen.hash3(seed, 1, ctr), n_cols), vals


@pytest.mark.parametrize("order", ["grouped", "any"])
@pytest.mark.parametrize("n_rows,n_cols,hubs", [
    (900, 5000, [(0, 12_285)]),                              # 12 288 entries: still a block's
    (900, 5000, [(0, 12_286)]),                              # one more, on few columns
    (900, (1 << 32) - 5, [(899, 20_000)]),                   # the widest columns, the last row
    (900, 1, [(450, 30_000)]),                               # one column: one entry is left
    (3000, 400_000, [(0, 15_000), (1, 13_000), (2500, 40_961), (2999, 12_286)]),
    (40, 70_000, [(r, 13_000 + r) for r in range(40)]),      # nothing but such rows
])
def test_lock_rows_longer_than_a_block(ctx, n_rows, n_cols, hubs, order):
    """Rows above 12 288 entries are sorted apart and put between the others,
    in a first lock and in a later one (whose zeros delete)."""
    epochs = []
    for seed in (1, 2):
        e = _hub_inserts(n_rows, n_cols, hubs, seed)
        if order == "any":
            p = np.argsort(gen.hash3(seed, 3, np.arange(len(e[0]), dtype=np.uint64)), kind="stable")
            e = tuple(x[p] for x in e)
        epochs.append(e)
    A = sg.Csr(ctx, n_rows, n_cols)
    for k in (1, 2):
        A.lock(*epochs[k - 1])
        assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, n_cols, epochs[:k]))


def test_lock_hub_row_among_clustered_rows(ctx):
    """More than the few-inserts rule, short rows of near columns (the row
    classes' case) and one row that they cannot take."""
    n = 1_100_000
    rows = np.repeat(np.arange(n, dtype=np.uint32), 4)
    ctr = np.arange(len(rows), dtype=np.uint64)
    cols = ((rows + gen.hash3(8, 1, ctr) % np.uint64(6)) % np.uint64(n)).astype(np.uint32)
    hub = np.full(13_000, 77, np.uint32)
    k = np.arange(len(hub), dtype=np.uint64)
    e = (np.insert(rows, 77 * 4, hub), np.insert(cols, 77 * 4, gen.below(gen.hash3(8, 2, k), n)),
         gen.sym_unit(gen.hash3(8, 3, np.arange(len(rows) + len(hub), dtype=np.uint64))))
    A = sg.Csr(ctx, n, n)
    A.lock(*e)
    assert_csr_equal(A.download(), oracle.lock_epochs(n, n, [e]))


@pytest.mark.parametrize("L", [33, 40, 2048, 2049, 4097, 12_288])
@pytest.mark.parametrize("wide", [False, True])
def test_lock_rows_of_more_inserts_than_columns(ctx, L, wide):
    """Rows around the point where each column of the row's range has a place
    of its own (range below length - 2), beside rows that are short or spread;
    the last write of a column wins, and a last zero leaves nothing."""
    n_cols = (1 << 31) + 7 if wide else 40_000
    lens, lo, rng = [], [], []
    for k in (L - 1, L - 2, L - 3, L // 2, 1, 0, 7):  # columns in the range
        for length in (L, 5, 0, 33):
            lens.append(length)
            lo.append(3 + 11 * len(lens))
            rng.append(max(1, min(k if length == L else n_cols - 1000, n_cols - 1000)))
    lens, lo, rng = (np.asarray(x, np.int64) for x in (lens, lo, rng))
    rows = np.repeat(np.arange(len(lens), dtype=np.uint32), lens)
    ctr = np.arange(len(rows), dtype=np.uint64)
    cols = (lo[rows] + (gen.hash3(L, 1, ctr) % rng[rows].astype(np.uint64)).astype(np.int64)).astype(np.uint32)
    first = np.r_[True, rows[1:] != rows[:-1]]  # the ends of every range occur
    last = np.r_[rows[1:] != rows[:-1], True]
    cols[first] = lo[rows[first]]
    cols[last] = lo[rows[last]] + rng[rows[last]] - 1
    vals = gen.sym_unit(gen.hash3(L, 2, ctr))
    vals[::5] = 0.0
    e = (rows, cols, vals)
    A = sg.Csr(ctx, len(lens), n_cols)
    A.lock(*e)
    assert_csr_equal(A.download(), oracle.lock_epochs(len(lens), n_cols, [e]))
    A.lock(*(x[::-1].copy() for x in e))
    assert_csr_equal(A.download(), oracle.lock_epochs(len(lens), n_cols, [e, tuple(x[::-1].copy() for x in e)]))


@pytest.mark.parametrize("mean", [1535, 1536, 2399, 2400, 4096, 4097])
@pytest.mark.parametrize("n_cols", [1 << 14, (1 << 14) + 1])
def test_lock_mean_row_length_rule(ctx, mean, n_cols):
    """Means of inserts per row at the ends of the ranges that go to the row
    classes, with rows of other lengths among them."""
    n = 40
    lens = np.full(n, mean, np.int64)
    lens[::4] += 900  # (the mean stays)
    lens[1::4] -= 900
    rows = np.repeat(np.arange(n, dtype=np.uint32), lens)
    ctr = np.arange(len(rows), dtype=np.uint64)
    cols = gen.below(gen.hash3(mean, 1, ctr), n_cols)
    vals = gen.sym_unit(gen.hash3(mean, 2, ctr))
    vals[::9] = 0.0
    A = sg.Csr(ctx, n, n_cols)
    A.lock(rows, cols, vals)
    assert_csr_equal(A.download(), oracle.lock_epochs(n, n_cols, [(rows, cols, vals)]))


@pytest.mark.parametrize("repeats", [False, True])
@pytest.mark.parametrize("zeros", [False, True])
def test_later_epoch_in_order_of_long_rows(ctx, repeats, zeros):
    """An epoch already in (row, column) order, of rows above 12 288 inserts,
    into a matrix with and without stored zeros (whose deletes join it)."""
    n, n_cols, per = 6, 300_000, 20_000
    first = _hub_inserts(n, n_cols, [(r, 5000) for r in range(n)], 3)
    H = oracle.lock_epochs(n, n_cols, [first])
    A = sg.Csr(ctx, n, n_cols)
    if zeros:
        v = H.vals.copy()
        v[::5] = 0.0
        A.load(H.off, H.cols, v)
        rows_of = np.repeat(np.arange(n, dtype=np.uint32), np.diff(H.off.astype(np.int64)))
        first = (rows_of[v != 0.0], H.cols[v != 0.0], v[v != 0.0])  # (zeros of dirty rows go away)
    else:
        A.lock(*first)
    r = np.repeat(np.arange(n, dtype=np.uint32), per)
    c = np.sort(gen.below(gen.hash3(4, 1, np.arange(len(r), dtype=np.uint64)), n_cols).reshape(n, per), axis=1)
    if not repeats:
        c = (np.arange(per, dtype=np.uint32) * 14 + np.arange(n, dtype=np.uint32)[:, None]).astype(np.uint32)
    v = gen.sym_unit(gen.hash3(4, 2, np.arange(len(r), dtype=np.uint64)))
    v[::9] = 0.0
    e = (r, c.reshape(-1).astype(np.uint32), v)
    A.lock(*e)
    assert_csr_equal(A.download(), oracle.lock_epochs(n, n_cols, [first, e]), check_capacity=not zeros)


@pytest.mark.parametrize("order", ["any", "streams"])
@pytest.mark.parametrize("n_rows,hubs,others", [
    (3000, 5, 0), (3000, 5, 20_000), (3000, 1, 90_000), (3000, 1, 300_000), (8, 8, 0), (40, 40, 2000),
])
def test_lock_unordered_with_hub_rows(ctx, n_rows, hubs, others, order):
    """Unordered inserts with some to all of them in rows of more than a block
    takes, in a first and a later lock: what the sample says changes the way, not
    the result. Streams: three ordered ones, one after another."""
    n_cols, epochs = 50_000, []
    for seed in (5, 6):
        m = hubs * 13_000 + others
        ctr = np.arange(m, dtype=np.uint64)
        r = np.where(ctr < hubs * 13_000, (ctr % np.uint64(hubs)) * np.uint64(max(1, n_rows // hubs)),
                     gen.hash3(seed, 1, ctr) % np.uint64(n_rows)).astype(np.uint32)
        p = np.argsort(gen.hash3(seed, 2, ctr), kind="stable")
        if order == "streams":
            p = np.concatenate([q[np.argsort(r[q], kind="stable")] for q in np.array_split(p, 3)])
        v = gen.sym_unit(gen.hash3(seed, 4, ctr))
        v[::8] = 0.0
        epochs.append((r[p], gen.below(gen.hash3(seed, 3, ctr), n_cols)[p], v[p]))
    A = sg.Csr(ctx, n_rows, n_cols)
    for k in (1, 2):
        A.lock(*epochs[k - 1])
        assert_csr_equal(A.download(), oracle.lock_epochs(n_rows, n_cols, epochs[:k]))
