"""The slice-pair product's plans: arenas that force column blocks, leading dimensions above the sizes, and the sum
inside the product kernel with three and four digits, against other paths of the same bits."""
import numpy as np
import pytest

from tests.conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu


def _dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a)).cuda()


def _phi(rng, shape, phi=1.0):
    return (rng.random(shape) - 0.5) * np.exp(phi * rng.standard_normal(shape))


@pytest.mark.parametrize("sm", [0, 1])
@pytest.mark.parametrize("m,n,k,digits,tile", [(700, 1200, 128, 4, 64), (500, 1800, 1024, 3, 96)])
def test_column_blocks(sm, m, n, k, digits, tile, handle, ozb, cuda):
    """Arenas that hold the digit planes and from one tile of the pair buffer's columns to all of them: every one is
    enough, for two blocks of whole tiles (the plan for 16 pairs of these sizes) or as many as it takes."""
    rng = np.random.default_rng(7)
    dA, dB = _dev(cuda, _phi(rng, (m, k))), _dev(cuda, _phi(rng, (n, k)))

    def run(h):
        h.sumMode = sm
        dC = cuda.zeros((n, m), dtype=cuda.float64, device="cuda")
        before = h.launch_count()
        ozb.dgemm(h, "t", "n", m, n, k, 1.0, dA, k, dB, k, 0.0, dC, m)
        return dC, h.launch_count() - before

    ref, launches = run(handle)
    assert handle.nSplitC == 16 and launches == 2 + 2 * 2  # two splits; products and sum per block
    planes = 0  # eight levels of digits, their exponents and the tiles' level counts, each from a 256-byte boundary
    for lines, t in ((m, 128), (n, tile)):
        for b in (8 * digits * lines * k, 16 * lines, 4 * -(-lines // t)):
            planes = -(-planes // 256) * 256 + b
    planes = -(-planes // 256) * 256
    half = -(-n // 2)
    for cols in (tile, tile + 1, n // 3, half - 1, half + 4, half + tile, n):
        h = ozb.Handle(work_bytes=planes + cols * 8 * 16 * m)
        out, launches = run(h)
        h.close()
        block = min(-(-half // tile), cols // tile) * tile
        assert launches == 2 + 2 * -(-n // block), cols
        assert cuda.equal(out, ref), cols


@pytest.mark.parametrize("form,ta,tb,m,n,k,mode", [
    ("d", "n", "t", 200, 150, 300, 0), ("d", "t", "n", 130, 300, 128, 0), ("d", "n", "n", 2100, 1700, 200, 0),
    ("d", "t", "n", 1300, 1100, 128, 0), ("d", "n", "t", 2100, 1700, 90, 0), ("d", "t", "t", 1, 300, 200, 0),
    ("sd", "n", "t", 200, 150, 300, 0), ("sd", "t", "n", 2100, 1700, 129, 0), ("sd", "n", "n", 1100, 900, 70000, 9)])
def test_leading_dimensions(form, ta, tb, m, n, k, mode, handle, ozb, cuda, monkeypatch):
    """lda, ldb and ldc above the sizes, a few lines that need more levels than the rest; the memory between the lines
    is NaN and stays so in C.  The last case has four digits in the mixed form."""
    gen = cuda.Generator(device="cuda").manual_seed(m + n + k)
    dt = cuda.float64 if form == "d" else cuda.float32

    def mat(lines, length, pad):
        full = cuda.full((lines, length + pad), float("nan"), dtype=dt, device="cuda")
        u = cuda.rand((lines, length), dtype=cuda.float64, device="cuda", generator=gen) - 0.5
        full[:, :length] = (u * cuda.randn((lines, length), dtype=cuda.float64, device="cuda", generator=gen).exp()).to(dt)
        return full

    A = mat(k, m, 5) if ta == "n" else mat(m, k, 3)
    B = mat(n, k, 1) if tb == "n" else mat(k, n, 2)
    if ta == "t" and m > 3:
        A[3, :k] *= cuda.exp2(cuda.randint(-40, 40, (k,), device="cuda", generator=gen).to(dt))
    C0 = mat(n, m, 7)
    handle.splitEpsMode = mode
    call = ozb.dgemm if form == "d" else ozb.sdgemm
    outs = []
    for dmma in (False, True):
        if dmma:
            monkeypatch.setenv("OZBLAS_PLAIN_DMMA" if form == "d" else "OZBLAS_SD_DMMA", "1")
            handle.read_env()
        C = C0.clone()
        call(handle, ta, tb, m, n, k, 1.25, A, A.shape[1], B, B.shape[1], -0.5, C, C.shape[1])
        outs.append(C.cpu().numpy())
    got, want = (o[:, :m].astype(np.float64) for o in outs)
    assert bits_equal(got, want), first_diff(got, want)
    assert np.isnan(outs[0][:, m:]).all()
