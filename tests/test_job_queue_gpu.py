"""The GEMM's scheduler warp (short inner dimensions, at least eight jobs per CTA): batches of 32 jobs that end
before, at and after a CTA's last job, bit for bit against the oracle, and its bounded waits, made to run out as in
the test of the kernel without it: the MMA issuer issues nothing, so every role gives up after a few milliseconds, the
call reports a timeout and the next one is exact."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu
WAIT_NS = 5_000_000


@pytest.fixture
def config(oz):
    yield oz.set_gemm_config
    oz.set_gemm_config(0, 16, 0)


def product(oz, A, B, C0, s):
    import torch
    dC = to_dev(C0)
    (m, k), n = A.shape, B.shape[1]
    oz.gemm("N", "N", m, n, k, 1.0, to_dev(A), m, to_dev(B), k, 0.5, dC, m, s)
    torch.cuda.synchronize()
    return dC


def expected(oracle, A, B, C0, s):
    (m, k), n = A.shape, B.shape[1]
    want = C0.copy(order="F")
    assert oracle.dgemm("N", "N", m, n, k, 1.0, A, m, B, k, 0.5, want, m, s) == 0
    return want


# jobs = s ceil(m / bn) ceil(n / 128), in CTAs of 8 (one batch), 31, 32, 33, 64, 65 and 96 (three batches) jobs
@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("s,cols,ctas", [(8, 1, 1), (8, 31, 8), (8, 4, 1), (11, 3, 1), (16, 4, 1), (13, 5, 1), (16, 6, 1),
                                         (13, 15, 3)])
def test_batches(oracle, oz, config, bn, s, cols, ctas):
    m, n, k = bn - 3, 128 * cols - 5, 40
    A, B, C0 = make_mat(s, m, k, m, "u"), make_mat(cols, k, n, k, "u"), make_mat(7, m, n, m, "u")
    config(bn, 16, ctas)
    got = from_dev(product(oz, A, B, C0, s), C0)
    oz.check_device_error()
    assert np.array_equal(bits(got), bits(expected(oracle, A, B, C0, s)))


@pytest.mark.parametrize("bn", [128, 256])
def test_stalled_queue_reports_timeout_and_the_next_call_is_exact(oracle, oz, config, bn):
    import oz2
    m, n, k, s = 640, 384, 256, 16  # 72 (256-row tiles) or 120 jobs per CTA: the scheduler waits for its third batch
    A, B, C0 = make_mat(901, m, k, m, "u"), make_mat(902, k, n, k, "u"), make_mat(903, m, n, m, "u")
    config(bn, 16, 2)
    oz.check_device_error()  # nothing pending before the test
    try:
        oz2.set_failure_test(WAIT_NS, stall_mma=True)
        product(oz, A, B, C0, s)
    finally:
        oz2.set_failure_test()
    with pytest.raises(TimeoutError):
        oz.check_device_error()
    want = expected(oracle, A, B, C0, s)
    for _ in range(2):
        got = from_dev(product(oz, A, B, C0, s), C0)
        oz.check_device_error()
        assert np.array_equal(bits(got), bits(want))
