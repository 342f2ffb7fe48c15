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
