"""The one-launch split of a short vector (GEMV's x) against the oracle, bit for bit: lengths at the edges of its forms,
and vectors whose largest element or largest remainder is subnormal, where tau depends on every bit of it."""
import numpy as np
import pytest

from oracle.oracle import make_flags
from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _vector(k, kind, seed):
    rng = np.random.default_rng(seed)
    x = (rng.random(k) - 0.5) * np.exp(rng.standard_normal(k))
    if kind == "phi":
        return x
    # odd multiples of 2^-1058: a grid of 2^-1057 or above rounds them
    x = (2 * rng.integers(-2 ** 20, 2 ** 20, k) + 1).astype(float) * 2.0 ** -1058
    if kind == "power":  # a power of two below the normal range: bits of its high word alone
        x[k // 2] = 2.0 ** -1034
    if kind == "above":  # just above one by the low word, far enough for the next tau
        x[k // 2] = np.uint64(0x0000100080000000).view(np.float64)
    if kind == "remainder":  # the first level leaves such a power
        x = np.where(rng.random(k) < 0.5, -1.0, 1.0) * 2.0 ** -1010
        x[k // 2] += 2.0 ** -1034
        x[k // 3] -= 3 * 2.0 ** -1058
    return x


@pytest.mark.parametrize("trans", ["n", "t"])
@pytest.mark.parametrize("k,kind", [(2048, "phi"), (2049, "phi"), (8192, "phi"), (8193, "phi"), (16384, "phi"),
                                    (64, "power"), (2049, "power"), (8193, "power"), (64, "above"), (64, "remainder")])
def test_dgemv_short_x(k, kind, trans, oracle, handle, ozb, cuda):
    nl = 9
    x = _vector(k, kind, k)
    lines = np.random.default_rng(1).standard_normal((nl, k))
    if kind != "phi":
        lines *= 2.0 ** 900
    A = lines if trans == "t" else np.ascontiguousarray(lines.T)  # rows of the array are columns of A
    m, n = (k, nl) if trans == "t" else (nl, k)
    y0 = np.arange(nl) * 2.0 ** (-160 if kind != "phi" else 0)
    ref, info = oracle.dgemv(make_flags(), trans, m, n, 0.75, A, m, x, 0.5, y0)

    def dev(a):
        return cuda.from_numpy(np.ascontiguousarray(a)).cuda()

    dy = dev(y0)
    ozb.dgemv(handle, trans, m, n, 0.75, dev(A), m, dev(x), 0.5, dy)
    assert (handle.nSplitA, handle.nSplitB) == (info.nSplitA, info.nSplitB)
    assert bits_equal(dy.cpu().numpy(), ref), first_diff(dy.cpu().numpy(), ref)
