"""ROWMERGE's choice between a thread's merge per row and the hash rows, and
AUTO's for rows of few products. Every way gives the same bits."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _matrix(ctx, n, per_row, near):
    rows = np.repeat(np.arange(n, dtype=np.uint32), per_row)
    ctr = np.arange(len(rows), dtype=np.uint64)
    if near:
        cols = ((rows.astype(np.uint64) + ctr % np.uint64(per_row)) % np.uint64(n)).astype(np.uint32)
    else:
        cols = gen.below(gen.hash3(n, 1, ctr), n)
    vals = np.where(gen.hash3(n, 2, ctr) % np.uint64(3) == 0, -1.0, 1.0)  # sums that cancel
    vals[::1001] = np.nan
    A = sg.Csr(ctx, n, n)
    A.lock(rows, cols, vals)
    return A, A.download()


@pytest.mark.parametrize("n,per_row,near", [
    (353_000, 1, False), (355_000, 1, False),  # hash rows, merge: where the rule turns
    (401_000, 2, True), (600_000, 3, True), (560_000, 3, False),
])
def test_rowmerge_of_many_short_rows(ctx, n, per_row, near):
    A, H = _matrix(ctx, n, per_row, near)
    want = oracle.spgemm(H, H)
    for v in (sg.SPGEMM_VARIANTS["rowmerge"], sg.SPGEMM_VARIANTS["warpsort_64"], -1):
        assert_csr_equal(A.spgemm(A, v).download(), want)


@pytest.mark.parametrize("n,per_row", [(10_000, 2), (100_000, 2), (1_000_000, 2), (1_000_000, 1)])
def test_auto_leaves_esc_to_long_rows(ctx, n, per_row):
    A, _ = _matrix(ctx, n, per_row, False)
    picked = A.spgemm_selected(A)
    assert picked in (sg.SPGEMM_VARIANTS["rowmerge"], sg.SPGEMM_VARIANTS["warpsort_64"])
    if n == 1_000_000:
        assert picked == sg.SPGEMM_VARIANTS["rowmerge"]
