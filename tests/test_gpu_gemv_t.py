"""GEMV 't' with the split and the slice products in registers against the path that materialises the slices, bit for
bit in both sum modes: line lengths at the edges of the staged chunks and of the warps per line, few and many lines,
lines whose remainders fall below the predicted chain, zero lines, infinities, long lines and truncated splits."""
import numpy as np
import pytest

from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _run(ozb, cuda, handle, A, k, nl, x, y0):
    dy = cuda.from_numpy(y0.copy()).cuda()
    ozb.dgemv(handle, "t", k, nl, 0.75, cuda.from_numpy(A).cuda(), A.shape[1], cuda.from_numpy(x).cuda(), 0.5, dy)
    return dy.cpu().numpy(), (handle.nSplitA, handle.nSplitB, handle.nSplitC)


@pytest.mark.parametrize("sm", [0, 1])
@pytest.mark.parametrize("k,nl,kind", [(1, 5, "phi"), (33, 200, "phi"), (256, 3000, "phi"), (513, 1201, "phi"),
                                       (2047, 37, "phi"), (6001, 301, "phi"), (16384, 9, "phi"), (16385, 9, "phi"),
                                       (700, 300, "close"), (3000, 64, "close"), (400, 90, "wide"),
                                       (500, 80, "zeros"), (300, 40, "inf"), (900, 50, "scaled")])
def test_dgemv_t_equals_materialised(sm, k, nl, kind, handle, ozb, cuda, monkeypatch):
    rng = np.random.default_rng(k + nl)
    lda = k + 3
    A = (rng.random((nl, lda)) - 0.5) * np.exp(rng.standard_normal((nl, lda)))
    x = (rng.random(k) - 0.5) * np.exp(rng.standard_normal(k))
    if kind == "close":  # remainders after level 0 far below the predicted chain
        A[::2] = 1.0 + 2.0 ** -45 * rng.choice([-1.0, 1.0], size=A[::2].shape)
    if kind == "wide":  # more levels than are held on chip
        A[7] *= np.exp2(rng.integers(-120, 120, lda).astype(float))
    if kind == "zeros":
        A[3] = 0.0
        x[::2] = 0.0
    if kind == "inf":
        A[5, 7] = np.inf
    if kind == "scaled":
        A *= 2.0 ** -600
        x *= 2.0 ** -450
    y0 = rng.standard_normal(nl)
    handle.sumMode = sm
    for nsplit in (0, 2):
        handle.nSplitMax = nsplit
        monkeypatch.delenv("OZBLAS_GEMV_SPLIT", raising=False)
        handle.read_env()
        got, ginfo = _run(ozb, cuda, handle, A, k, nl, x, y0)
        monkeypatch.setenv("OZBLAS_GEMV_SPLIT", "1")
        handle.read_env()
        ref, rinfo = _run(ozb, cuda, handle, A, k, nl, x, y0)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert bits_equal(np.nan_to_num(got), np.nan_to_num(ref)), first_diff(got, ref)
        assert ginfo == rinfo
