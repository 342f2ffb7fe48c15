"""Transpose of matrices with 16 to 32 entries a column on average: rows that
repeat each other's pattern are sorted by the networks, others by the column
sort, also where the sample is wrong. Bit-exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _csr(n, m, per_row, kind):
    rows = np.repeat(np.arange(n, dtype=np.uint32), per_row)
    k = np.tile(np.arange(per_row, dtype=np.uint64), n)
    if kind == "band":
        cols = (rows + k) % m
    elif kind == "blocks":
        cols = (rows // per_row * per_row + k) % m
    elif kind == "hub":  # a band, and one column in every row
        cols = np.where(k == 0, 0, (rows + k) % m)
    else:
        cols = gen.below(gen.hash3(n, 1, np.arange(len(rows), dtype=np.uint64)), m)
    vals = gen.sym_unit(gen.hash3(n, 2, np.arange(len(rows), dtype=np.uint64)))
    return oracle.lock_epochs(n, m, [(rows, cols.astype(np.uint32), vals)])


@pytest.mark.parametrize("kind", ["band", "blocks", "hub", "uniform"])
@pytest.mark.parametrize("n,m,per_row", [(2, 2, 2), (1, 40, 40), (40, 1, 1), (700, 700, 17), (4097, 4097, 32),
                                         (5000, 5000, 33), (60_000, 60_000, 17), (60_000, 60_000, 18),
                                         (70_000, 70_000, 32), (70_000, 70_000, 33), (90_000, 45_000, 12)])
def test_transpose_by_sample(ctx, n, m, per_row, kind):
    H = _csr(n, m, per_row, kind)
    A = sg.Csr(ctx, n, m)
    A.load(H.off, H.cols, H.vals)
    assert_csr_equal(A.transpose().download(), oracle.transpose(H))


@pytest.mark.parametrize("kind", ["band", "uniform"])
def test_transpose_of_many_entries(ctx, kind):
    H = _csr(620_000, 620_000, 17, kind)  # above 10 M entries
    A = sg.Csr(ctx, H.n_rows, H.n_cols)
    A.load(H.off, H.cols, H.vals)
    assert_csr_equal(A.transpose().download(), oracle.transpose(H))
