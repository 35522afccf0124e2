"""The slice-pair product's plans, against other paths of the same bits."""
import numpy as np
import pytest

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
