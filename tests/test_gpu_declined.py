"""What a call pays when a short form cannot hold its input: the launches and the time reported are those of the path
that computes the result."""
import numpy as np
import pytest

from oracle.oracle import make_flags

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sm", [0, 1])
@pytest.mark.parametrize("n,kind", [(1000, "deep"), (4096, "deep"), (600, "inf"), (600, "nan")])
def test_short_dot_beyond_one_launch(sm, n, kind, handle, ozb, cuda, monkeypatch):
    """More than 8 levels, Inf or NaN: the two-pass forms cannot hold them either, so one declined launch is all that is
    added to the general path."""
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    if kind == "deep":
        x *= 2.0 ** rng.integers(-120, 120, n)
    else:
        x[n // 2] = np.inf if kind == "inf" else np.nan
    dx, dy = cuda.from_numpy(x).cuda(), cuda.from_numpy(y).cuda()
    handle.sumMode = sm

    def run():
        before = handle.launch_count()
        r = ozb.ddot(handle, n, dx, dy)
        return np.float64(r).view(np.int64), handle.launch_count() - before

    got, launches = run()
    monkeypatch.setenv("OZBLAS_DOT_TREE", "1")  # scan and product pass (2 launches), declined, then the general path
    monkeypatch.setenv("OZBLAS_DOT_TWO_PASS", "1")
    handle.read_env()
    want, before = run()
    assert got == want
    assert launches == before - 1


@pytest.mark.parametrize("kx,ky,kind", [(950, -400, ""), (-980, 500, ""), (-1030, 900, ""), (505, 480, ""), (-500, -440, "")])
@pytest.mark.parametrize("sm", [0, 1])
def test_short_dot_at_range_ends(sm, kx, ky, kind, oracle, handle, ozb, cuda):
    """Sigmas, grids and products near the ends of the range that the one launch holds."""
    n = 300
    rng = np.random.default_rng(n)
    x, y = rng.integers(-2 ** 30, 2 ** 30, n) * 2.0 ** -30, rng.integers(-2 ** 30, 2 ** 30, n) * 2.0 ** -30
    x, y = np.ldexp(x, kx), np.ldexp(y, ky)
    handle.sumMode = sm
    before = handle.launch_count()
    r = ozb.ddot(handle, n, cuda.from_numpy(x).cuda(), cuda.from_numpy(y).cuda())
    assert handle.launch_count() - before == 1
    ref, info = oracle.ddot(make_flags(sumMode=sm), x, y)
    assert np.float64(r).view(np.int64) == np.float64(ref).view(np.int64), (r, ref)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)


def test_csrmv_general_path_time(handle, ozb, cuda):
    """x off the predicted chain: t_comp spans the general path's kernels, not those of the path that declined."""
    n, w = 400000, 6
    gen = cuda.Generator(device="cuda").manual_seed(1)
    rowptr = cuda.arange(0, (n + 1) * w, w, dtype=cuda.int32, device="cuda")
    colind = cuda.randint(0, n, (n * w,), dtype=cuda.int32, device="cuda", generator=gen)
    val = cuda.randn(n * w, dtype=cuda.float64, device="cuda", generator=gen)
    x = cuda.randn(n, dtype=cuda.float64, device="cuda", generator=gen) * 2.0 ** -40
    x[n // 2] = 1.0
    y = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    for _ in range(3):
        ozb.dcsrmv(handle, "n", n, n, n * w, 1.0, val, colind, rowptr, x, 0.0, y)
    # the declined path: 3 kernels of some 100 us; the general one: count, write, split of x and products
    cuda.cuda.synchronize()
    assert handle.t_comp > 0.5 * handle.t_total, (handle.t_comp, handle.t_total)
