"""The long FSum DOT on the INT8 tensor cores against the FP64 tree pass, bit for bit: two and three digits per level,
few and all levels, lengths that end inside a job and leave groups of a block without one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("n,phi", [(1 << 22, 0.5), ((1 << 22) + 1, 1.0), ((1 << 22) + 1023, 3.0), (5000001, 0.0),
                                   ((1 << 24) + 7, 1.0)])
def test_ddot_i8_equals_tree(n, phi, same, handle, ozb, cuda, monkeypatch):
    gen = cuda.Generator(device="cuda").manual_seed(n)
    x = (cuda.rand(n, dtype=cuda.float64, device="cuda", generator=gen) - 0.5) * cuda.exp(
        phi * cuda.randn(n, dtype=cuda.float64, device="cuda", generator=gen))
    y = x if same else cuda.flip(x, [0]).contiguous() * 3.0
    got = ozb.ddot(handle, n, x, y), handle.nSplitA, handle.nSplitB
    monkeypatch.setenv("OZBLAS_DOT_TREE", "1")
    handle.read_env()
    want = ozb.ddot(handle, n, x, y), handle.nSplitA, handle.nSplitB
    assert np.float64(got[0]).view(np.int64) == np.float64(want[0]).view(np.int64) and got[1:] == want[1:], (got, want)
