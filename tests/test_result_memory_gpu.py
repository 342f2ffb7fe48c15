"""Results of A + B and of ROWMERGE's hash rows hold about their own size, also
where the sample that sizes their arrays is wrong. Bit-exact against the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu
SAMPLES, ROW_SAMPLES = 1024, 2048


def _held(ctx, make):
    """(result, device bytes that it added)."""
    make().close()
    ctx.sync()
    before = ctx.pool_used()[0]
    C = make()
    ctx.sync()
    return C, ctx.pool_used()[0] - before


def _own_size(C):
    i = C.info()
    return 12 * i["nnz"] + 8 * (i["n_rows"] + 1)


def _load(ctx, H):
    A = sg.Csr(ctx, H.n_rows, H.n_cols)
    A.load(H.off, H.cols, H.vals)
    return A


def _rows_of(n, per_row, seed, n_cols):
    """per_row ascending columns per row, an even step apart."""
    step = n_cols // per_row
    r = np.repeat(np.arange(n, dtype=np.uint32), per_row)
    k = np.tile(np.arange(per_row, dtype=np.uint64), n)
    c = (k * np.uint64(step) + gen.hash3(seed, 1, np.arange(len(r), dtype=np.uint64)) % np.uint64(step)).astype(np.uint32)
    return oracle.lock_epochs(n, n_cols, [(r, c, gen.sym_unit(gen.hash3(seed, 2, np.arange(len(r), dtype=np.uint64))))])


@pytest.mark.parametrize("case", ["same", "other", "cancel", "misleading", "few"])
def test_add_holds_its_own_size(ctx, case):
    n, per = (250_000, 10) if case != "few" else (2000, 10)
    H = _rows_of(n, per, 1, 1_000_000)
    A = _load(ctx, H)
    if case in ("same", "few"):
        HB = H
    elif case == "cancel":
        HB = oracle.lock_epochs(n, H.n_cols, [(np.repeat(np.arange(n, dtype=np.uint32), per), H.cols, -H.vals)])
    elif case == "other":
        HB = _rows_of(n, per, 2, 1_000_000)
    else:  # every sampled entry of the larger side is in the other, hardly any else
        k = np.arange(SAMPLES, dtype=np.uint64)
        part = np.uint64(len(H.cols) // SAMPLES)
        e = (part * k + (k * np.uint64(0x9E3779B1) >> np.uint64(8)) % part).astype(np.int64)
        rows = np.repeat(np.arange(n, dtype=np.uint32), per)
        o = _rows_of(n, per - 1, 3, 1_000_000)
        HB = oracle.lock_epochs(n, H.n_cols, [(np.concatenate([np.repeat(np.arange(n, dtype=np.uint32), per - 1), rows[e]]),
                                               np.concatenate([o.cols, H.cols[e]]),
                                               np.concatenate([o.vals, np.ones(SAMPLES)]))])
        assert len(HB.cols) < len(H.cols)
    B = _load(ctx, HB)
    C, held = _held(ctx, lambda: A.add(B))
    assert_csr_equal(C.download(), oracle.add(H, HB))
    if case != "few":
        assert held <= 1.15 * _own_size(C) + (1 << 20)


@pytest.mark.parametrize("case", ["collapsing", "distinct", "misleading"])
def test_hash_rows_hold_their_own_size(ctx, case):
    """100 k rows of 8 times 8 products."""
    m, groups, width = 100_000, 4096, 500_000
    k = np.arange(ROW_SAMPLES, dtype=np.uint64)
    part = np.uint64(m // ROW_SAMPLES)
    sampled = (k * part + (k * np.uint64(0x9E3779B1) >> np.uint64(8)) % part).astype(np.int64)
    collapse = np.zeros(m, bool)
    collapse[:] = case == "collapsing"
    if case == "misleading":
        collapse[sampled] = True
    r = np.repeat(np.arange(m, dtype=np.uint32), 8)
    j = np.tile(np.arange(8, dtype=np.uint32), m)
    # B's rows: 0..7 have the same eight columns, the others columns of their own
    ac = np.where(collapse[r], j, 8 + (r * 7 + j * 131) % (groups - 8)).astype(np.uint32)
    HA = oracle.lock_epochs(m, groups, [(r, ac, gen.sym_unit(gen.hash3(1, 1, np.arange(len(r), dtype=np.uint64))))])
    br = np.repeat(np.arange(groups, dtype=np.uint32), 8)
    bj = np.tile(np.arange(8, dtype=np.uint32), groups)
    bc = np.where(br < 8, bj * 1000, (br * 97 + bj * 60_013) % width).astype(np.uint32)
    HB = oracle.lock_epochs(groups, width, [(br, bc, gen.sym_unit(gen.hash3(1, 2, np.arange(len(br), dtype=np.uint64))))])
    A, B = _load(ctx, HA), _load(ctx, HB)
    C, held = _held(ctx, lambda: A.spgemm(B, sg.SPGEMM_VARIANTS["rowmerge"]))
    assert_csr_equal(C.download(), oracle.spgemm(HA, HB))
    assert held <= 1.15 * _own_size(C) + (1 << 20)
