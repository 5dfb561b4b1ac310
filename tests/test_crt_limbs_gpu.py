"""The CRT above eight 16-bit limbs, bit for bit against the oracle: complex operands at every number of moduli that
keeps 24 residue planes (s = 17..24), and the extended sets of the adaptive path (13 to 16 limbs, s = 26..32) at the
edges of the 32-row by 16-column tiles and for results far below the largest the plan allows."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev
from test_crt_gpu import SIZES, cancelling, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", range(17, 25))
def test_zgemm(oracle, oz, s):
    for q, (m, n) in enumerate(SIZES):
        A, B = make_mat(3 * s + q, m, 20, m, "wide", 12, cplx=True), make_mat(5 * s + q, 20, n, 20, "wide", 12, cplx=True)
        check(oracle, oz, A, B, make_mat(q, m, n, m + q % 3, "u", cplx=True), s, 1.0 + 0.5j, 0.25 - 1.0j if q % 2 else 0.0)


def check_extended(oracle, oz, A, B, C0, s, alpha=1.0, beta=0.0):
    import torch
    (m, k), n, ldc = A.shape, B.shape[1], C0.shape[0]
    dC = to_dev(C0)
    oz.gemm_adaptive([("N", "N", m, n, k, alpha, to_dev(A), m, to_dev(B), k, beta, dC, ldc, s)], 53, oz.ADAPTIVE_FIXED)
    torch.cuda.synchronize()
    oz.check_device_error()
    want = C0.copy(order="F")
    assert oracle.dgemm_ext("N", "N", m, n, k, alpha, A, m, B, k, beta, want, ldc, s) == 0
    got = from_dev(dC, C0)
    assert np.array_equal(bits(got), bits(want)), f"{int((bits(got) != bits(want)).sum())} words differ"


@pytest.mark.parametrize("s", [25, 26, 28, 30, 31, 32])
def test_extended_sizes(oracle, oz, s):
    for q, (m, n) in enumerate(SIZES):
        A, B = make_mat(100 * s + q, m, 40, m, "wide", 30), make_mat(200 * s + q, 40, n, 40, "wide", 30)
        check_extended(oracle, oz, A, B, make_mat(300 + q, m, n, m + q % 3, "u"), s, 1.5, -0.5 if q % 2 else 0.0)


@pytest.mark.parametrize("s", [25, 26, 28, 30, 32])
def test_extended_results_far_below_the_plan(oracle, oz, s):
    tails = np.array([0.0, 1.0, -1.0, 2.0, -2.0, 2.0 ** 24, -(2.0 ** 24), 2.0 ** 24 - 1, 3.0])
    A, B, X, Y = cancelling(40, 40, tails)
    B[0], B[1] = Y, -X  # row i, column i: X Y - Y X + tail
    check_extended(oracle, oz, A, B, np.zeros((40, 40), order="F"), s)
