"""GEMV 't' with lines beyond the levels held in registers, or with infinities and NaN, which a block each follows level
by level, and with x beyond them (the slice path, with x's slices kept): against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _case(kind, nl, k):
    rng = np.random.default_rng(nl + k)
    A = (rng.random((nl, k)) - 0.5) * np.exp(rng.standard_normal((nl, k)))
    x = (rng.random(k) - 0.5) * np.exp(rng.standard_normal(k))
    deep = np.exp2(rng.integers(-110, 110, k).astype(float))
    if kind in ("some", "zeros in x", "no x"):
        A[1::3] *= deep
        A[2] = 0.0
    if kind == "all":
        A *= deep
    if kind == "few bits":  # many levels predicted; one in truth, or seven
        A[0] = np.where(rng.random(k) < 0.5, 1.0, 2.0 ** -250)
        A[1, :] = 0.0
        A[1, :7] = np.exp2(-40.0 * np.arange(7))
    if kind == "nonfinite":
        A[0, 3], A[4, k - 1], A[nl - 1, 0] = np.inf, np.nan, -np.inf
        A[2] *= deep
    if kind == "ends":  # grids below the range that the kernels take
        A[1] *= deep * 2.0 ** -880
    if kind == "x":
        x *= deep
    if kind == "zeros in x":
        x[::2] = 0.0
    if kind == "no x":
        x[:] = 0.0
    return A, x, rng.standard_normal(nl)


@pytest.mark.parametrize("sm,nsplit", [(0, 0), (1, 0), (0, 3), (0, 9)])
@pytest.mark.parametrize("nl,k,kind", [(7, 300, "some"), (100, 513, "all"), (5, 16384, "all"), (40, 255, "few bits"),
                                       (33, 700, "nonfinite"), (20, 400, "ends"), (50, 600, "x"),
                                       (30, 320, "zeros in x"), (9, 100, "no x"), (6, 1, "some")])
def test_dgemv_t_deep(nl, k, kind, sm, nsplit, oracle, handle, ozb, cuda):
    A, x, y0 = _case(kind, nl, k)
    ref, info = oracle.dgemv(make_flags(sumMode=sm, nSplitMax=nsplit), "t", k, nl, 0.75, A, k, x, 0.5, y0)
    handle.sumMode, handle.nSplitMax = sm, nsplit
    dA, dx, dy = (cuda.from_numpy(v.copy()).cuda() for v in (A, x, y0))
    ozb.dgemv(handle, "t", k, nl, 0.75, dA, k, dx, 0.5, dy)
    out = dy.cpu().numpy()
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    assert bits_equal(np.nan_to_num(out), np.nan_to_num(ref)), first_diff(out, ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)


def test_dgemv_t_deep_launches(handle, ozb, cuda):
    """One line beyond the levels held: x's split, statistics, products and y, then that line and y again."""
    A, x, y0 = _case("some", 4, 1000)
    dA, dx, dy = (cuda.from_numpy(v.copy()).cuda() for v in (A, x, y0))
    before = handle.launch_count()
    ozb.dgemv(handle, "t", 1000, 4, 0.75, dA, 1000, dx, 0.5, dy)
    assert handle.launch_count() - before == 6


@pytest.mark.parametrize("kind", ["x", "ends"])
def test_dgemv_t_slice_path_small_arena(kind, handle, ozb, cuda):
    """Arenas that hold the slice path's own buffers but not x's kept slices beside them."""
    nl, k = 64, 1000
    A, x, y0 = _case(kind, nl, k)
    dA, dx = (cuda.from_numpy(v.copy()).cuda() for v in (A, x))

    def run(h):
        dy = cuda.from_numpy(y0.copy()).cuda()
        ozb.dgemv(h, "t", k, nl, 0.75, dA, k, dx, 0.5, dy)
        return dy

    ref = run(handle)
    # nA slices of A, 30 of x, and twice the pair products
    nA, nB = int(handle.nSplitA), int(handle.nSplitB)
    need = 8 * (nA * nl * k + 30 * k + 2 * nA * nB * nl) + 8192
    for extra in (0, 100_000, 20_000_000):
        h = ozb.Handle(work_bytes=need + extra)
        assert cuda.equal(run(h), ref)
        h.close()
