"""Failure detection without a GPU fault: each kind of wait between blocks, run
against a predecessor that never publishes, gives up after its limit, writes
nothing and leaves the context usable."""
from __future__ import annotations

import ctypes as C

import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu

KINDS = {"scan": 1, "block": 2, "row_sort": 4}


@pytest.mark.parametrize("wait_cycles", [1, 200_000, 20_000_000])
def test_every_wait_gives_up_and_context_stays_usable(wait_cycles):
    ctx = sg.Context(0)
    kinds = C.c_int(0)
    sg._check(sg.lib().spg_selftest_wait_kinds(ctx.h, wait_cycles, C.byref(kinds)))
    assert kinds.value == sum(KINDS.values())
    with pytest.raises(sg.DeviceTimeout):
        ctx.sync()
    ctx.sync()  # reported once, then cleared
    n = 3000
    r, c, v = (x[::-1].copy() for x in gen.uniform_rows(n, n, 6, seed=2))
    A = sg.Csr(ctx, n, n)
    A.lock(r, c, v)
    H = oracle.lock_epochs(n, n, [(r, c, v)])
    assert_csr_equal(A.download(), H)
    assert_csr_equal(A.add(A).download(), oracle.add(H, H))
    assert_csr_equal(A.spgemm(A, sg.SPGEMM_VARIANTS["rowmerge"]).download(), oracle.spgemm(H, H))
    ctx.close()
