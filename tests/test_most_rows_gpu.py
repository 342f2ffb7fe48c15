"""A later lock() of a matrix of 2^32 rows (the transpose of one of 2^32
columns): the last tile of rows ends at 2^32, which no 32-bit row number
holds. Takes about 170 GB of device memory, in a process of its own so that
the memory goes back."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
N = 1 << 32


def _run(order):
    import spira_gb300 as sg

    ctx = sg.Context(0)
    first = np.array([0, 1, 5, 4096, 2 ** 31, N - 2049, N - 2, N - 1] + list(range(7000, 7022)), np.uint32)
    A = sg.Csr(ctx, 1, N)
    A.lock(np.zeros(len(first), np.uint32), first, np.arange(1.0, len(first) + 1.0))
    T = A.transpose()
    assert T.n_rows == N
    # above a fifth of the matrix: not insert by insert. Overwrites, new rows, deletes, a row written twice
    rows = np.array([0, 3, 3, 4096, 7000, 2 ** 31 + 1, N - 2048, N - 3, N - 1, N - 1], np.uint32)
    vals = np.array([-1.0, 0.0, -2.0, 0.0, -3.0, -4.0, -5.0, -6.0, 0.0, -7.0])
    if order == "any":
        p = np.array([4, 1, 8, 0, 5, 2, 7, 9, 3, 6])  # (the second write of a row stays after the first)
        rows, vals = rows[p], vals[p]
    assert len(rows) > T.nnz // 5
    T.lock(rows, np.zeros(len(rows), np.uint32), vals)
    want = dict(zip(first.tolist(), np.arange(1.0, len(first) + 1.0).tolist()))
    want.update(zip(rows.tolist(), vals.tolist()))
    want = {r: v for r, v in sorted(want.items()) if v != 0.0}
    assert T.row_range(N - 1) == (len(want) - 1, len(want))
    back = T.transpose().download()
    np.testing.assert_array_equal(back.off, np.array([0, len(want)], np.uint64))
    np.testing.assert_array_equal(back.cols, np.array(list(want), np.uint32))
    np.testing.assert_array_equal(back.vals, np.array(list(want.values())))


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["grouped", "any"])
def test_relock_of_2_to_32_rows(order):
    import torch

    if torch.cuda.mem_get_info()[0] < 200 << 30:
        pytest.skip("needs 200 GB of free device memory")
    code = f"import sys; sys.path[:0] = [{str(ROOT)!r}, {str(ROOT / 'tests')!r}]; import {Path(__file__).stem} as t; t._run({order!r})"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
