"""The CRT at the edges of its tiles and at the edges of its rounding, bit for bit against the oracle.

Tiles: 32 rows by 8 warps of 4 columns (up to 16 moduli) or 2 columns (more moduli, or complex).
Rounding: results far below the largest the plan allows (whole top words that only repeat the sign),
exact zeros, ties to even, integers around powers of two, subnormal results and overflow.
"""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu


def check(oracle, oz, A, B, C0, s, alpha=1.0, beta=0.0):
    import torch
    m, k = A.shape
    n = B.shape[1]
    cplx = np.iscomplexobj(A)
    dC = to_dev(C0)
    ldc = C0.shape[0]
    call = oz.zgemm if cplx else oz.gemm
    call("N", "N", m, n, k, alpha, to_dev(A), m, to_dev(B), k, beta, dC, ldc, s)
    torch.cuda.synchronize()
    oz.check_device_error()
    want = C0.copy(order="F")
    ref = oracle.zgemm if cplx else oracle.dgemm
    assert ref("N", "N", m, n, k, alpha, A, m, B, k, beta, want, ldc, s) == 0
    got = from_dev(dC, C0)
    assert np.array_equal(bits(got), bits(want)), f"{int((bits(got) != bits(want)).sum())} words differ"


SIZES = [(1, 1), (7, 9), (31, 5), (32, 16), (33, 3), (64, 33), (65, 17), (100, 301)]


@pytest.mark.parametrize("s", [2, 3, 5, 7, 9, 12, 14, 16, 17, 19, 21, 24])
def test_dgemm_sizes(oracle, oz, s):
    for q, (m, n) in enumerate(SIZES):
        k = 5 if s < 5 else 40
        A, B = make_mat(100 * s + q, m, k, m, "wide", 3), make_mat(200 * s + q, k, n, k, "wide", 3)
        check(oracle, oz, A, B, make_mat(300 + q, m, n, m + q % 3, "u"), s, 1.5, -0.5 if q % 2 else 0.0)


@pytest.mark.parametrize("s", [5, 8, 13, 16, 18, 24])
def test_zgemm_sizes(oracle, oz, s):
    for q, (m, n) in enumerate(SIZES):
        A, B = make_mat(7 * s + q, m, 20, m, "u", cplx=True), make_mat(9 * s + q, 20, n, 20, "u", cplx=True)
        check(oracle, oz, A, B, make_mat(q, m, n, m + q % 3, "u", cplx=True), s, 1.0 + 0.5j, 0.25 - 1.0j if q % 2 else 0.0)


def cancelling(rows, cols, tails):
    """A and B whose products are the small integers tails[i]: two terms X Y - Y X of 2 x 25 bits cancel"""
    rng = np.random.default_rng(5)
    X, Y = rng.integers(1 << 24, 1 << 25, (2, rows)).astype(float)
    A = np.zeros((rows, 3), order="F")
    A[:, 0], A[:, 1], A[:, 2] = X, Y, np.resize(tails, rows)
    B = np.zeros((3, cols), order="F")
    B[2] = 1.0
    return A, B, X, Y


@pytest.mark.parametrize("s", [10, 13, 16, 20, 24])
def test_results_far_below_the_plan(oracle, oz, s):
    tails = np.array([0.0, 1.0, -1.0, 2.0, -2.0, 2.0 ** 24, -(2.0 ** 24), 2.0 ** 24 - 1, 3.0])
    A, B, X, Y = cancelling(40, 40, tails)
    B[0], B[1] = Y, -X  # row i, column i: X Y - Y X + tail
    check(oracle, oz, A, B, np.zeros((40, 40), order="F"), s)


@pytest.mark.parametrize("s", [14, 16, 18, 24])
def test_ties_and_powers_of_two(oracle, oz, s):
    p = np.array([2.0 ** 53, 2.0 ** 53 - 1, 2.0 ** 52, 2.0 ** 52 - 1, 2.0 ** 31, 2.0 ** 32, 2.0 ** 47])
    d = np.array([0.0, 1.0, -1.0, 2.0, 3.0, 0.5, -0.5, 0.25])
    A = np.asfortranarray(np.column_stack([np.repeat(p, len(d)), np.tile(d, len(p))]))
    B = np.asfortranarray(np.array([[1.0, -1.0, 1.0, 2.0 ** 40, -3.0], [1.0, -1.0, -1.0, 2.0 ** 40, 1.0]]))
    check(oracle, oz, A, B, np.zeros((A.shape[0], 5), order="F"), s)


@pytest.mark.parametrize("ea,eb", [(-600, -450), (-540, -534), (500, 520), (-1000, 0)])
def test_subnormal_results_and_overflow(oracle, oz, ea, eb):
    A = np.ldexp(make_mat(1, 33, 6, 33, "wide", 20), ea)
    B = np.ldexp(make_mat(2, 6, 9, 6, "wide", 20), eb)
    for s in (12, 16, 22):
        check(oracle, oz, np.asfortranarray(A), np.asfortranarray(B), np.zeros((33, 9), order="F"), s)
