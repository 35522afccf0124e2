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


@pytest.mark.parametrize("n,kind", [(1, ""), (33, ""), (1024, ""), (1025, "rising"), (40001, "rising"),
                                    (40001, "blocks"), (5000, "cancel"), (3000, "zeros"), (70000, "high"),
                                    (70000, "low")])
def test_exact_reduction_bins(n, kind, oracle, handle, ozb, cuda):
    x, y = oracle.phi_vector(n, 1.0, 1), oracle.phi_vector(n, 1.0, 2)
    if kind == "rising":
        x *= 2.0 ** np.linspace(-30, 30, n).astype(int)
    if kind == "blocks":
        x *= np.where((np.arange(n) // 1024) % 3 == 0, 2.0 ** 50, 2.0 ** -20)
    if kind == "cancel":
        x[n // 2:], y[n // 2:] = x[:n - n // 2], -y[:n - n // 2]
    if kind == "zeros":
        x[::2] = 0.0
    if kind in ("high", "low"):
        x *= 2.0 ** (400 if kind == "high" else -400)
    handle.sumMode = 1
    dx, dy = cuda.from_numpy(x).cuda(), cuda.from_numpy(y).cuda()
    d = ozb.ddot(handle, n, dx, dy)
    r, info = oracle.ddot(make_flags(sumMode=1), x, y)
    assert np.float64(d).view(np.int64) == np.float64(r).view(np.int64), (d, r)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
