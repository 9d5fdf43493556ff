"""Rows per stage group at widths where rows made longer for tensor copies would
leave a stage fewer of them: a group keeps at least three quarters of the rows
that fit 96 KB as they are, 19 directions each (at most 8)."""
import re

import pytest

import dnslbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,nx", [(64, 90), (64, 92), (64, 209), (64, 212), (32, 181), (32, 417), (32, 428), (32, 641),
                                     (32, 644), (16, 353), (16, 833), (16, 848), (64, 628), (32, 402)])
def test_longer_rows_keep_the_groups(prec, nx, monkeypatch):
    for e in ("ROW_ALIGN", "GROUP_ROWS", "STAGES"):
        monkeypatch.delenv("DNSLBM_" + e, raising=False)
    size = prec // 8
    align = 16 if size == 4 else 32
    row = (nx * size + align - 1) // align * align
    fit = min(8, 98304 // (19 * row))
    with dnslbm.Channel(nx, 40, 8, 1.7, gx=1e-5, precision=prec) as ch:
        rows = int(re.search(r"groups of (\d+) rows", ch.kernel).group(1))
    assert 4 * rows >= 3 * fit and rows <= fit
