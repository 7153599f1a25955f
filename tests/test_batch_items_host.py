"""Rows per item of a batch (no GPU): a register chain's items outweigh the
rows that precede them, staged kernels keep their four or 64 rows."""

from types import SimpleNamespace

import pytest

from cutile.runtime.rk_runtime import batch_zchunk
from cutile.runtime.serving import batch_zchunk as served_zchunk


@pytest.mark.parametrize("T,rz", [(2, 1), (5, 1), (8, 1)])
def test_chain_items_outweigh_their_lead(T, rz):
    """T steps of skew and the T rz rows above an item come before its first
    row (four-row items made a batch of FP64 chains three times slower)."""
    d = {"rows": 1, "threads": 128, "nslot": 0, "temporal": T, "rz": T * rz, "zchunk": -8}
    assert served_zchunk is batch_zchunk
    assert batch_zchunk(SimpleNamespace(desc=d)) >= T * rz + T


@pytest.mark.parametrize("zchunk,rows", [(-8, 32), (0, 64), (16, 64)])
def test_staged_kernels_are_unchanged(zchunk, rows):
    d = {"rows": 8, "threads": 128, "nslot": 3, "temporal": 1, "rz": 1, "zchunk": zchunk}
    assert batch_zchunk(SimpleNamespace(desc=d)) == rows
