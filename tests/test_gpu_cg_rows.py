"""Rows and reductions of the sparse and NearSum paths against the oracle, bit for bit: CG over matrices whose rows are
all fit for the flat row kernel and over ones that are not (long, deep, zero-sum rows), the row split at every lane
width, and the exact reductions with bins that start high, rise and differ between blocks."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _sym(n, deg, seed):
    """A symmetric, diagonally dominant matrix with at most `deg` entries in a row, as (rowptr, colind, val)."""
    rng = np.random.default_rng(seed)
    rows = [{i: 0.0} for i in range(n)]
    for _ in range(4 * n):
        i, j = (int(v) for v in rng.integers(0, n, 2))
        if i != j and len(rows[i]) < deg and len(rows[j]) < deg:
            rows[i][j] = rows[j][i] = float(rng.random() - 0.5)
    for i in range(n):
        rows[i][i] = 1.0 + sum(abs(v) for v in rows[i].values()) + float(rng.random())
    rowptr = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    colind = np.concatenate([sorted(r) for r in rows]).astype(np.int32)
    val = np.concatenate([[r[c] for c in sorted(r)] for r in rows])
    return rowptr, colind, val


@pytest.mark.parametrize("n,deg,kind", [(1, 1, ""), (255, 7, ""), (256, 8, ""), (257, 8, ""), (1500, 5, ""),
                                        (700, 12, ""), (600, 6, "deep"), (600, 6, "integers"), (300, 6, "huge")])
def test_cg_rows(n, deg, kind, oracle, handle, ozb, cuda):
    rowptr, colind, val = _sym(n, deg, n + deg)
    b = oracle.normal(n, 4)
    if kind == "deep":  # one row needs more levels than the others
        val[rowptr[n // 2]] *= 2.0 ** -70
    if kind == "integers":  # row sums that cancel to zero, midpoints
        val, b = np.rint(val * 4), np.rint(b * 2)
    if kind == "huge":  # products near the top of the range
        val, b = val * 2.0 ** 500, b * 2.0 ** 400
    iters = 5
    xr, hr, _ = oracle.dcg(make_flags(sumMode=1), val, colind, rowptr, b, np.zeros(n), iters, 0.0)
    handle.sumMode, handle.verbose = 1, 1

    def dev(a):
        return cuda.from_numpy(np.ascontiguousarray(a)).cuda()

    dx = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    h1, h2 = np.zeros(iters + 1), np.zeros(iters + 1)
    ozb.dcg(handle, "n", n, len(val), dev(val), dev(colind), dev(rowptr), dev(b), dx, iters, 0.0, h1, h2)
    assert bits_equal(h1, hr), first_diff(h1, hr)
    assert bits_equal(dx.cpu().numpy(), xr), first_diff(dx.cpu().numpy(), xr)


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


@pytest.mark.parametrize("sm", [0, 1])
def test_many_deferred_rows(sm, oracle, handle, ozb, cuda):
    """More rows of over 8 entries than one launch with terms in memory takes, some with sums that need NearSum itself."""
    rng = np.random.default_rng(3)
    n = 20000
    lens = np.where(np.arange(n) % 2 == 0, 10, 3)
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colind = rng.integers(0, n, int(rowptr[-1])).astype(np.int32)
    val = oracle.phi_vector(len(colind), 1.0, 7)
    x, y0 = oracle.phi_vector(n, 1.0, 8), oracle.phi_vector(n, 1.0, 9)
    for r in range(0, n, 40):  # entries that cancel in pairs: zero sums, which the certified sum leaves to NearSum
        lo = rowptr[r]
        colind[lo + 5:lo + 10] = colind[lo:lo + 5]
        val[lo + 5:lo + 10] = -val[lo:lo + 5]
    ref, info = oracle.dcsrmv(make_flags(sumMode=sm), n, n, 0.5, val, colind, rowptr, x, -2.0, y0)

    def dev(a):
        return cuda.from_numpy(np.ascontiguousarray(a)).cuda()

    handle.sumMode = sm
    dy = dev(y0)
    ozb.dcsrmv(handle, "n", n, n, len(val), 0.5, dev(val), dev(colind), dev(rowptr), dev(x), -2.0, dy)
    assert bits_equal(dy.cpu().numpy(), ref), first_diff(dy.cpu().numpy(), ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
