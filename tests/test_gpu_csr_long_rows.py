"""The CSR row split with a few rows far longer than the rest, one or many, scattered or together (the last case: more
of them in one block than it lists), against the oracle."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sm", [0, 1])
@pytest.mark.parametrize("n,short,long_rows", [(2000, 2, {700: 1999}), (3000, 3, {0: 17, 1: 16, 2: 15, 2999: 3000}),
                                               (1500, 1, {r: 900 for r in range(600, 640)}),
                                               (4000, 6, {r: 40 + r % 7 for r in range(0, 4000, 100)}),
                                               (700, 0, {5: 700, 6: 600}), (9000, 80, {4: 8192, 5: 8193, 8999: 9000}),
                                               (700000, 3, {148 * 8 * 128 * i + j: 40 for i in range(4) for j in range(128)}
                                                | {148 * 8 * 512 + j: 41 for j in range(128)})])
def test_long_rows(sm, n, short, long_rows, oracle, handle, ozb, cuda):
    """x off the predicted chain, so that the rows' slices come from the row split."""
    rng = np.random.default_rng(n)
    lens = rng.integers(0, short + 1, n)
    for r, l in long_rows.items():
        lens[r] = min(l, n)
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colind = rng.integers(0, n, int(rowptr[-1])).astype(np.int32)
    val = oracle.phi_vector(len(colind), 1.0, 7)
    for r in long_rows:  # the long rows need more levels than the others
        val[rowptr[r]] *= 2.0 ** -60
    x, y0 = oracle.phi_vector(n, 1.0, 8) * 2.0 ** -40, oracle.phi_vector(n, 1.0, 9)
    x[n // 2] = 1.0
    flags = make_flags(sumMode=sm)
    ref, info = oracle.dcsrmv(flags, n, n, 0.5, val, colind, rowptr, x, -2.0, y0)

    def dev(a):
        return cuda.from_numpy(np.ascontiguousarray(a)).cuda()

    handle.sumMode = sm
    dval, dcol, drow = dev(val), dev(colind), dev(rowptr)
    dy = dev(y0)
    ozb.dcsrmv(handle, "n", n, n, len(val), 0.5, dval, dcol, drow, dev(x), -2.0, dy)
    assert bits_equal(dy.cpu().numpy(), ref), first_diff(dy.cpu().numpy(), ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
    ns, shift, _ = oracle.dcsrmv_split_a(flags, val, rowptr)
    ozb.dcsrmv_split_a(handle, "n", n, n, len(val), dval, drow)
    assert (handle.nSplitA_, handle.splitShift) == (ns, shift)
    handle.memMaskSplitA = 0


def test_one_long_row_in_time(handle, ozb, cuda):
    """A third of the entries in one row: the split takes a small multiple of the time it takes without that row (it
    was hundreds of times in the row's own few lanes)."""
    m = 100000
    times = []
    for length in (3, 150000):
        lens = cuda.full((m,), 3, dtype=cuda.int64, device="cuda")
        lens[m // 2] = length
        rowptr = cuda.zeros(m + 1, dtype=cuda.int64, device="cuda")
        rowptr[1:] = cuda.cumsum(lens, 0)
        nnz, rowptr = int(rowptr[-1]), rowptr.int()
        val = cuda.randn(nnz, dtype=cuda.float64, device="cuda", generator=cuda.Generator("cuda").manual_seed(1))
        best = 1e9
        for _ in range(4):
            handle.memMaskSplitA = 0
            ozb.dcsrmv_split_a(handle, "n", m, m, nnz, val, rowptr)
            best = min(best, handle.t_total)
        times.append(best)
    handle.memMaskSplitA = 0
    assert times[1] < 20 * times[0], times
