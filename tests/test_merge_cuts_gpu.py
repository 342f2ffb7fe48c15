"""The CSR merge (spira_gb300/csrc/spg_merge.cu) with its tiles of 1020 items
(entries of both sides and row ends) cut at and around row ends, and through
rows of one entry on either side or of an equal pair."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import spira_gb300 as sg
from spira_gb300 import gen
from conftest import assert_csr_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [339, 340, 341, 509, 510, 511, 1019, 1020, 1021, 3061])
@pytest.mark.parametrize("a,b,equal", [(0, 0, False), (1, 0, False), (1, 1, True), (1, 1, False), (2, 1, True), (1020, 3, True)])
def test_merge_at_the_tiles_cuts(ctx, n, a, b, equal):
    """a and b entries a row: 1, 2, 3, 4 or more items, which divide the tile or
    do not; the pair of an equal column is never cut apart."""
    def rows(per, off):
        r = np.repeat(np.arange(n, dtype=np.uint32), per)
        c = (np.tile(np.arange(per, dtype=np.uint32) * 2, n) + off).astype(np.uint32)
        return r, c, gen.sym_unit(gen.hash3(n, per + off, np.arange(len(r), dtype=np.uint64)))

    if a == 1020:
        n = min(n, 40)
    ea, eb = rows(a, 0), rows(b, 0 if equal else 1)
    Ha, Hb = oracle.lock_epochs(n, 3000, [ea]), oracle.lock_epochs(n, 3000, [eb])
    A, B = sg.Csr(ctx, n, 3000), sg.Csr(ctx, n, 3000)
    A.lock(*ea)
    B.lock(*eb)
    assert_csr_equal(A.add(B).download(), oracle.add(Ha, Hb))
    assert_csr_equal(B.add(A).download(), oracle.add(Hb, Ha))
    if b:
        A.lock(*eb)
        assert_csr_equal(A.download(), oracle.lock_epochs(n, 3000, [ea, eb]))
