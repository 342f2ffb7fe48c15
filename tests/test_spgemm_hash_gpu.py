"""ROWMERGE's hash rows (spira_gb300/csrc/spg_spgemm_hash.cu): at most 64
products per row, eight lanes a row, tiles of 32 rows. Full tables, all
products on one column, exact cancellations, B rows of one to 64 entries, A
rows of one to 64 entries, ragged last tiles; one product more sends every row
the other way. Bit-exact against the oracle's order without contraction."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


def _matrix(n_rows, n_cols, lengths, seed, spread):
    rows = np.repeat(np.arange(n_rows, dtype=np.uint32), lengths)
    first = np.cumsum(lengths) - lengths
    k = np.arange(len(rows)) - np.repeat(first, lengths)
    # distinct columns per row: a start and a step
    start = gen.below(gen.hash3(seed, 1, np.arange(n_rows, dtype=np.uint64)), n_cols).astype(np.int64)
    cols = ((np.repeat(start, lengths) + k * spread) % n_cols).astype(np.uint32)
    vals = gen.sym_unit(gen.hash3(seed, 2, np.arange(len(rows), dtype=np.uint64)))
    vals[::3] = 1.0   # sums that cancel exactly
    vals[1::3] = -1.0
    return oracle.lock_epochs(n_rows, n_cols, [(rows, cols, vals)])


def _dev(ctx, H):
    A = sg.Csr(ctx, H.n_rows, H.n_cols)
    A.load(H.off, H.cols, H.vals)
    return A


@pytest.mark.parametrize("m", [1, 31, 32, 33, 5000])
@pytest.mark.parametrize("a_len,b_len", [(1, 64), (64, 1), (8, 8), (7, 9), (9, 7), (2, 32), (5, 13)])
@pytest.mark.parametrize("spread", [1, 97])
def test_rowmerge_hash_rows(ctx, m, a_len, b_len, spread):
    kdim, n = 300, 40_000
    h = gen.hash3(m, 5, np.arange(m, dtype=np.uint64))
    la = np.where(h % np.uint64(4) == 0, (h >> np.uint64(8)) % np.uint64(a_len + 1), a_len).astype(np.int64)
    lb = np.full(kdim, b_len, np.int64)
    lb[::7] = b_len // 2
    A, B = _matrix(m, kdim, la, 3, 1), _matrix(kdim, n, lb, 4, spread)
    got = _dev(ctx, A).spgemm(_dev(ctx, B), sg.SPGEMM_VARIANTS["rowmerge"]).download()
    assert_csr_equal(got, oracle.spgemm(A, B))


def test_rowmerge_one_product_too_many(ctx):
    A, B = _matrix(200, 300, np.full(200, 5, np.int64), 3, 1), _matrix(300, 500, np.full(300, 13, np.int64), 4, 3)
    assert oracle.spgemm_products(A, B) == 200 * 65
    got = _dev(ctx, A).spgemm(_dev(ctx, B), sg.SPGEMM_VARIANTS["rowmerge"]).download()
    assert_csr_equal(got, oracle.spgemm(A, B))
