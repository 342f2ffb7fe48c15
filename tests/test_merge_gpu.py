"""The tiled merge of two CSRs (spira_gb300/csrc/spg_merge.cu) behind A + B and
the later locks: cuts inside long rows and between equal columns, one side
empty or far denser than the other, long stretches of empty rows, deletes.
Bit-exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _epoch(lengths, n_cols, seed, zero_every=0):
    rows = np.repeat(np.arange(len(lengths), dtype=np.uint32), lengths)
    ctr = np.arange(len(rows), dtype=np.uint64)
    cols = gen.below(gen.hash3(seed, 1, ctr), n_cols)
    vals = gen.sym_unit(gen.hash3(seed, 2, ctr))
    vals[::97] = np.nan
    if zero_every:
        vals[::zero_every] = 0.0
    return rows, cols, vals


def _lengths(kind, n):
    h = gen.hash3(n, 7, np.arange(n, dtype=np.uint64))
    L = (h % np.uint64(6)).astype(np.int64)
    if kind == "long":  # rows of many tiles among short ones
        L[:: max(1, n // 5)] = 9000
    elif kind == "empty":
        L[:] = 0
        L[n // 2] = 3
    elif kind == "dense":
        L += 40
    return L


@pytest.mark.parametrize("n", [1, 2, 2039, 2040, 2041, 20_000])
@pytest.mark.parametrize("a,b", [("short", "short"), ("long", "long"), ("long", "short"), ("dense", "empty"),
                                 ("empty", "long"), ("empty", "empty")])
def test_merge_add_and_relock(ctx, n, a, b):
    n_cols = 15_000
    ea = _epoch(_lengths(a, n), n_cols, seed=1)
    eb = _epoch(_lengths(b, n), n_cols, seed=2, zero_every=5)
    back = (eb[0][::-1].copy(), eb[1][::-1].copy(), eb[2][::-1].copy())  # the delta in no order
    Ah, Bh = oracle.lock_epochs(n, n_cols, [ea]), oracle.lock_epochs(n, n_cols, [eb])
    A, B = sg.Csr(ctx, n, n_cols), sg.Csr(ctx, n, n_cols)
    A.lock(*ea)
    B.lock(*eb)
    assert_csr_equal(A.add(B).download(), oracle.add(Ah, Bh))
    assert_csr_equal(B.add(A).download(), oracle.add(Bh, Ah))
    assert_csr_equal(A.add(A).download(), oracle.add(Ah, Ah))
    half = tuple(x[::2].copy() for x in ea)  # overwrites and deletes of what is there
    half[2][::3] = 0.0
    for second in (back, half):
        C = sg.Csr(ctx, n, n_cols)
        C.lock(*ea)
        C.lock(*second)
        assert_csr_equal(C.download(), oracle.lock_epochs(n, n_cols, [ea, second]))
