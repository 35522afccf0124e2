"""Rows and reductions of the sparse and NearSum paths against the oracle, bit for bit: CG over matrices whose rows are
all fit for the flat row kernel and over ones that are not (long, deep, zero-sum rows), the row split at every lane
width, and the exact reductions with bins that start high, rise and differ between blocks."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lo,hi", [(1, 1, 1), (3000, 0, 2), (700, 1, 7), (500, 0, 40), (300, 20, 40), (200, 30, 199)])
def test_row_split_widths(n, lo, hi, oracle, handle, ozb, cuda):
    """x off the predicted chain: the rows' slices come from the row split, at each number of lanes per row."""
    rng = np.random.default_rng(n)
    lens = rng.integers(lo, hi + 1, n)
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colind = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lens]).astype(np.int32)
    val = oracle.phi_vector(len(colind), 1.0, 7)
    x, y0 = oracle.phi_vector(n, 1.0, 8) * 2.0 ** -40, oracle.phi_vector(n, 1.0, 9)
    x[n // 2] = 1.0
    ref, info = oracle.dcsrmv(make_flags(), n, n, 0.5, val, colind, rowptr, x, -2.0, y0)

    def dev(a):
        return cuda.from_numpy(np.ascontiguousarray(a)).cuda()

    dy = dev(y0)
    ozb.dcsrmv(handle, "n", n, n, len(val), 0.5, dev(val), dev(colind), dev(rowptr), dev(x), -2.0, dy)
    assert bits_equal(dy.cpu().numpy(), ref), first_diff(dy.cpu().numpy(), ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
