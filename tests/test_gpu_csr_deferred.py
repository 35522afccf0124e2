"""Rows of over 8 entries under NearSum, some with sums that only NearSum itself settles: one launch for as many rows as
have their terms in memory at once, against the oracle."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,launches", [(2000, 4), (8192, 4), (8193, 5)])
def test_deferred_rows_with_zero_sums(n, launches, oracle, handle, ozb, cuda):
    rng = np.random.default_rng(n)
    rowptr = np.arange(0, 10 * n + 1, 10).astype(np.int32)
    colind = rng.integers(0, n, 10 * n).astype(np.int32)
    val = oracle.phi_vector(10 * n, 1.0, 7)
    x, y0 = oracle.phi_vector(n, 1.0, 8), oracle.phi_vector(n, 1.0, 9)
    for r in range(0, n, 40):  # entries that cancel in pairs
        colind[10 * r + 5:10 * r + 10], val[10 * r + 5:10 * r + 10] = colind[10 * r:10 * r + 5], -val[10 * r:10 * r + 5]
    ref, info = oracle.dcsrmv(make_flags(sumMode=1), n, n, 0.5, val, colind, rowptr, x, -2.0, y0)
    handle.sumMode = 1
    dval, dcol, drow, dx, dy = (cuda.from_numpy(v.copy()).cuda() for v in (val, colind, rowptr, x, y0))
    before = handle.launch_count()
    ozb.dcsrmv(handle, "n", n, n, len(val), 0.5, dval, dcol, drow, dx, -2.0, dy)
    assert bits_equal(dy.cpu().numpy(), ref), first_diff(dy.cpu().numpy(), ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
    # x's statistics, its proof, the rows, the deferred ones (then those left open)
    assert handle.launch_count() - before == launches
