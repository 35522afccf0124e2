"""GEMV 'n' over rows of every state the passes tell apart (proven by the first pass or the second, left to the exact
passes, beyond the levels held), alone and mixed, on its three paths and against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _rows(kind, m, n, rng):
    """m rows of n elements."""
    R = (rng.random((m, n)) - 0.5) * np.exp(rng.standard_normal((m, n)))
    close = 1.0 + 2.0 ** -45 * rng.choice([-1.0, 1.0], size=(m, n))  # a remainder far below the predicted one
    gap = np.where(rng.random((m, n)) < 0.5, 1.0, 2.0 ** -250)  # many levels predicted, two in truth
    deep = R * np.exp2(rng.integers(-110, 110, (m, n)).astype(float))  # more levels than are held
    if kind == "close":
        R[::3] = close[::3]
    if kind == "gap":
        R[1::4] = gap[1::4]
    if kind == "all gap":
        R = gap
    if kind == "mixed":
        R[::3], R[1::5], R[7] = close[::3], gap[1::5], 0.0
    if kind == "deep":
        R[::40] = deep[::40]
        R[1::5] = gap[1::5]
    if kind == "all deep":
        R = deep
    if kind == "nan":
        R[5, 3], R[9] = np.nan, gap[9]
    return R


@pytest.mark.parametrize("sm,fm", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("m,n,kind", [(33, 100, "phi"), (300, 257, "close"), (200, 1000, "gap"), (64, 3000, "all gap"),
                                      (257, 700, "mixed"), (130, 513, "deep"), (96, 200, "all deep"), (40, 300, "nan")])
def test_dgemv_rows(m, n, kind, sm, fm, oracle, handle, ozb, cuda, monkeypatch):
    rng = np.random.default_rng(m + n)
    A = np.ascontiguousarray(_rows(kind, m, n, rng).T)  # rows of the array are columns of A
    x = (rng.random(n) - 0.5) * np.exp(rng.standard_normal(n))
    y0 = rng.standard_normal(m)
    ref, info = oracle.dgemv(make_flags(sumMode=sm, fastMode=fm), "n", m, n, 0.75, A, m, x, 0.5, y0)
    handle.sumMode, handle.fastMode = sm, fm
    monkeypatch.setenv("OZBLAS_GEMV_SLICES", "1")  # NearSum too by the slices
    dA, dx = cuda.from_numpy(A).cuda(), cuda.from_numpy(x).cuda()
    for env in (None, "OZBLAS_GEMV_LEVELS", "OZBLAS_GEMV_SPLIT"):
        if env:
            monkeypatch.setenv(env, "1")
        handle.read_env()
        dy = cuda.from_numpy(y0).cuda()
        ozb.dgemv(handle, "n", m, n, 0.75, dA, m, dx, 0.5, dy)
        out = dy.cpu().numpy()
        assert np.array_equal(np.isnan(out), np.isnan(ref)), env
        assert bits_equal(np.nan_to_num(out), np.nan_to_num(ref)), (env, first_diff(out, ref))
        assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB), env


def test_dgemv_deep_rows_passes(handle, ozb, cuda, monkeypatch):
    """Rows beyond the levels held: statistics, the passes over the chains, two sums that find a flag set, and nothing
    else before the path that materialises the slices."""
    m, n = 96, 400
    A = np.ascontiguousarray(_rows("all deep", m, n, np.random.default_rng(1)).T)
    dA, dx = cuda.from_numpy(A).cuda(), cuda.ones(n, dtype=cuda.float64, device="cuda")
    launches = []
    for env in (None, "OZBLAS_GEMV_SPLIT"):
        if env:
            monkeypatch.setenv(env, "1")
            handle.read_env()
        dy = cuda.zeros(m, dtype=cuda.float64, device="cuda")
        before = handle.launch_count()
        ozb.dgemv(handle, "n", m, n, 1.0, dA, m, dx, 0.0, dy)
        launches.append(handle.launch_count() - before)
    # x's split, statistics and chains, two fast and three exact passes with their checks, two sums
    assert launches[0] - launches[1] <= 1 + 2 + 2 * 5 + 2, launches
