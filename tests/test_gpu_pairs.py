"""The slice-pair products on the INT8 tensor cores (split into balanced int8 digits, all digit levels of a pair
accumulated in one pass, the ordered sum in the kernel or over a pair buffer) against the DMMA slice path: the pair
products are exact, so every bit agrees.  Sizes at the edges of the tiles (128 x 96, or 128 x 64 with four digits),
of the k steps and of the split's forms; rows that need more levels than the rest; infinities."""
import numpy as np
import pytest

from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _data(rng, shape, phi, wide):
    a = (rng.random(shape) - 0.5) * np.exp(phi * rng.standard_normal(shape))
    if wide:  # a few lines (both directions) spread over hundreds of bits, one zero line
        a[3] *= np.exp2(rng.integers(-150, 150, shape[1]).astype(float))
        a[:, 2] *= np.exp2(rng.integers(-40, 40, shape[0]).astype(float))
        a[4] = 0.0
    return a


CASES = [
    # m, n, k, ta, tb, sumMode, fastMode, wide
    (128, 96, 129, "n", "n", 0, 0, False),
    (129, 97, 128, "t", "t", 0, 0, False),
    (127, 95, 2048, "n", "t", 1, 0, True),
    (7, 300, 500, "t", "n", 0, 1, True),
    (300, 6, 2049, "n", "n", 0, 0, True),
    (385, 193, 40, "t", "n", 1, 1, False),
    (65, 64, 16385, "n", "n", 0, 0, False),
    (40, 33, 50000, "t", "n", 0, 0, False),
    (2100, 1700, 300, "n", "n", 0, 0, True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:3])) + f"-{c[3]}{c[4]}-s{c[5]}f{c[6]}")
@pytest.mark.parametrize("form", ["d", "sd"])
def test_pairs_equal_slice_path(form, case, handle, ozb, cuda, monkeypatch):
    m, n, k, ta, tb, sm, fm, wide = case
    if form == "sd" and sm == 1:
        pytest.skip("the mixed forms have no NearSum")
    rng = np.random.default_rng(m + 7 * n + k)
    A = _data(rng, (k, m) if ta == "n" else (m, k), 1.0, wide)
    B = _data(rng, (n, k) if tb == "n" else (k, n), 2.0, False)
    C0 = rng.standard_normal((n, m))
    if form == "sd":
        A, B, C0 = (np.clip(v, -1e30, 1e30).astype(np.float32) for v in (A, B, C0))
    dt, call = (np.float64, ozb.dgemm) if form == "d" else (np.float32, ozb.sdgemm)
    handle.sumMode, handle.fastMode = sm, fm
    dA, dB = (cuda.from_numpy(np.ascontiguousarray(v)).cuda() for v in (A, B))
    outs = []
    for dmma in (False, True):
        if dmma:
            monkeypatch.setenv("OZBLAS_PLAIN_DMMA" if form == "d" else "OZBLAS_SD_DMMA", "1")
            handle.read_env()
        dC = cuda.from_numpy(C0.astype(dt)).cuda()
        call(handle, ta, tb, m, n, k, 1.25, dA, m if ta == "n" else k, dB, k if tb == "n" else n, -0.5, dC, m)
        outs.append((dC.cpu().numpy().astype(np.float64), handle.nSplitA, handle.nSplitB, handle.nSplitC))
    assert bits_equal(outs[0][0], outs[1][0]), first_diff(outs[0][0], outs[1][0])
    assert outs[0][1:] == outs[1][1:]


def test_pairs_nonfinite(handle, ozb, cuda):
    """An infinity makes its row of the product NaN (its remainder is inf - inf) and touches nothing else."""
    rng = np.random.default_rng(3)
    m, n, k = 200, 150, 300
    A, B = _data(rng, (m, k), 1.0, False), _data(rng, (n, k), 1.0, False)
    outs = []
    for bad in (False, True):
        if bad:
            A[17, 5] = np.inf
            B[9, 250] = np.nan
        dC = cuda.zeros((n, m), dtype=cuda.float64, device="cuda")
        ozb.dgemm(handle, "t", "n", m, n, k, 1.0, cuda.from_numpy(A).cuda(), k, cuda.from_numpy(B).cuda(), k, 0.0, dC, m)
        outs.append(dC.cpu().numpy())
    hit = np.zeros((n, m), dtype=bool)
    hit[:, 17] = hit[9] = True
    assert np.array_equal(np.isnan(outs[1]), hit)
    assert bits_equal(outs[0][~hit], outs[1][~hit])
