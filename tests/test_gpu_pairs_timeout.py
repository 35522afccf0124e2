"""A bounded wait of the slice-pair product that runs out: the call reports it, C keeps its values where they go through
the pair buffer, and the next call on the handle gives its bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a)).cuda()


def _phi(rng, shape, phi=1.0):
    return (rng.random(shape) - 0.5) * np.exp(phi * rng.standard_normal(shape))


@pytest.mark.parametrize("form,m,n,sm", [("d", 300, 200, 0), ("d", 300, 200, 1), ("sd", 300, 200, 0), ("q", 150, 130, 0)])
def test_timeout_leaves_c(form, m, n, sm, oracle, handle, ozb, cuda):
    """Through the pair buffer: the producer holds back its copies and the waits are short, so the call returns
    DEVICE_TIMEOUT (6) with C as it was; restored, the same call gives its bits."""
    k = 300
    handle.sumMode = sm
    if form == "q":
        A, B, C0 = oracle.phi_matrix_q(k, m, 1.0, 1), oracle.phi_matrix_q(k, n, 1.0, 2), oracle.phi_matrix_q(m, n, 1.0, 3)
        A, B, C0 = (v.view(np.int64) for v in (A, B, C0))
        al, be, call = oracle.q(1.5), oracle.q(-0.5), ozb.qgemm
    else:
        rng = np.random.default_rng(5)
        dt = np.float64 if form == "d" else np.float32
        A, B, C0 = (_phi(rng, s).astype(dt) for s in ((m, k), (n, k), (n, m)))
        al, be, call = 1.5, -0.5, ozb.dgemm if form == "d" else ozb.sdgemm
    dA, dB = _dev(cuda, A), _dev(cuda, B)

    def run(dC):
        call(handle, "t", "n", m, n, k, al, dA, k, dB, k, be, dC, m)

    first, held, again = (_dev(cuda, C0) for _ in range(3))
    run(first)
    ozb.set_i8_wait_test(20_000_000, hold_copies=True)
    try:
        with pytest.raises(ozb.OzblasError) as e:
            run(held)
        assert e.value.code == 6
    finally:
        ozb.set_i8_wait_test(0, hold_copies=False)
    cuda.cuda.synchronize()
    run(again)
    assert np.array_equal(held.cpu().numpy(), C0)
    assert cuda.equal(again, first)


@pytest.mark.parametrize("m,n,k", [(2100, 1700, 300), (1300, 1100, 128)])
def test_timeout_in_fused_sum(m, n, k, handle, ozb, cuda):
    """With the sum inside the product kernel (CTAs that wait for one another's partial sums among them)."""
    rng = np.random.default_rng(6)
    dA, dB = _dev(cuda, _phi(rng, (m, k))), _dev(cuda, _phi(rng, (n, k)))

    def run():
        dC = cuda.zeros((n, m), dtype=cuda.float64, device="cuda")
        ozb.dgemm(handle, "t", "n", m, n, k, 1.0, dA, k, dB, k, 0.0, dC, m)
        return dC

    first = run()
    ozb.set_i8_wait_test(20_000_000, hold_copies=True)
    try:
        with pytest.raises(ozb.OzblasError) as e:
            run()
        assert e.value.code == 6
    finally:
        ozb.set_i8_wait_test(0, hold_copies=False)
    cuda.cuda.synchronize()
    assert cuda.equal(run(), first)
