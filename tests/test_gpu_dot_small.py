"""The one-launch DOT / NRM2 of short vectors against the other DOT paths, bit for bit in both sum modes: lengths at the
edges of the block and of its range, chains that are not the predicted one, zeros, truncated splits, and the inputs
that one launch leaves to the others (many levels, infinities, the ends of the range)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(v):
    return np.float64(v).view(np.int64)


@pytest.mark.parametrize("sm", [0, 1])
@pytest.mark.parametrize("n,kind,nsplit", [(1, "phi", 0), (2, "phi", 0), (255, "phi", 0), (256, "phi", 0),
                                           (257, "phi", 0), (1024, "phi", 0), (1025, "phi", 0), (4095, "phi", 0),
                                           (4096, "phi", 0), (4097, "phi", 0), (700, "close", 0), (300, "zeros", 0),
                                           (50, "allzero", 0), (500, "phi", 1), (1500, "phi", 2), (2000, "deep", 0),
                                           (600, "inf", 0), (600, "nan", 0), (400, "tiny", 0), (400, "huge", 0),
                                           (400, "subnormal", 0), (100, "powers", 0)])
def test_ddot_small_equals_other_paths(sm, n, kind, nsplit, handle, ozb, cuda, monkeypatch):
    rng = np.random.default_rng(n)
    x = (rng.random(n) - 0.5) * np.exp(rng.standard_normal(n))
    y = (rng.random(n) - 0.5) * np.exp(rng.standard_normal(n))
    if kind == "close":  # remainders after level 0 far below the predicted chain
        x = 1.0 + 2.0 ** -45 * rng.choice([-1.0, 1.0], n)
    if kind == "zeros":
        x[::3], y[::2] = 0.0, -0.0
    if kind == "allzero":
        x[:] = 0.0
    if kind == "deep":  # more than 8 levels
        x *= 2.0 ** rng.integers(-120, 120, n)
    if kind == "inf":
        x[n // 2] = np.inf
    if kind == "nan":
        y[n // 3] = np.nan
    if kind in ("tiny", "huge"):
        x, y = x * 2.0 ** (-500 if kind == "tiny" else 480), y * 2.0 ** (-490 if kind == "tiny" else 470)
    if kind == "subnormal":
        x *= 2.0 ** -1040
    if kind == "powers":
        x, y = 2.0 ** rng.integers(-20, 20, n), 2.0 ** rng.integers(-20, 20, n)
    dx, dy = cuda.from_numpy(x).cuda(), cuda.from_numpy(y).cuda()
    handle.sumMode, handle.nSplitMax = sm, nsplit

    def run():
        return [(_bits(ozb.ddot(handle, n, dx, dy)), handle.nSplitA, handle.nSplitB),
                (_bits(ozb.dnrm2(handle, n, dx)), handle.nSplitA, handle.nSplitB)]

    got = run()
    monkeypatch.setenv("OZBLAS_DOT_TREE", "1")
    monkeypatch.setenv("OZBLAS_DOT_TWO_PASS", "1")
    handle.read_env()
    want = run()
    assert got == want, (got, want)
