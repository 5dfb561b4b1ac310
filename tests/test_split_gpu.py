"""The split on the mma.sync byte products, at the edges of its tiles and of its copy paths.

Every result is compared bit for bit with the oracle: rows around the block tile (16, or 8 for
complex operands) and the 128-row plane tile, inner indices around 128, operands that are only
8-byte aligned (8-byte copies) or have odd leading dimensions, the three widths of the offset
integer, rows whose scaling takes two factors, and non-finite rows.
"""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, op_shape, to_dev

pytestmark = pytest.mark.gpu


def shifted(x, offset):
    """device copy of column-major `x` that starts `offset` doubles past an aligned address"""
    import torch
    flat = to_dev(x)
    buf = torch.empty(flat.numel() + offset, dtype=torch.float64, device="cuda")
    buf[offset:] = flat
    return buf[offset:]


CASES = [  # m, n, k, s, leading dimension pad, base offset in doubles
    (1, 1, 1, 8, 0, 0),
    (15, 17, 127, 13, 1, 0),
    (16, 33, 128, 14, 0, 1),
    (129, 127, 129, 16, 2, 0),
    (145, 8, 2305, 16, 0, 0),   # a span of 18 k blocks
    (31, 130, 255, 18, 1, 1),   # tk = 62..63: two or three words
    (64, 47, 384, 21, 4, 0),
    (257, 9, 130, 24, 1, 0),
]


@pytest.mark.parametrize("ops", ["NN", "TT", "TN"])
@pytest.mark.parametrize("case", CASES)
def test_dgemm_equals_the_oracle(oracle, oz, case, ops):
    import torch
    m, n, k, s, pad, off = case
    ta, tb = ops
    Ar, Ac = op_shape(ta, m, k)
    Br, Bc = op_shape(tb, k, n)
    A = make_mat(3 + s, Ar, Ac, Ar + pad, "wide", 12)
    B = make_mat(5 + s, Br, Bc, Br + pad, "wide", 12)
    C0 = make_mat(7 + s, m, n, m, "u")
    dC = to_dev(C0)
    oz.gemm(ta, tb, m, n, k, 1.5, shifted(A, off), A.shape[0], shifted(B, off), B.shape[0], -0.5, dC, m, s)
    torch.cuda.synchronize()
    want = C0.copy(order="F")
    assert oracle.dgemm(ta, tb, m, n, k, 1.5, A, A.shape[0], B, B.shape[0], -0.5, want, m, s) == 0
    assert np.array_equal(bits(from_dev(dC, C0)), bits(want))


@pytest.mark.parametrize("ops", ["NN", "CT", "TC"])
@pytest.mark.parametrize("case", [(7, 9, 127, 12, 0, 0), (8, 17, 129, 16, 1, 1), (130, 5, 300, 19, 0, 1), (33, 129, 64, 24, 1, 0)])
def test_zgemm_equals_the_oracle(oracle, oz, case, ops):
    import torch
    m, n, k, s, pad, off = case
    ta, tb = ops
    Ar, Ac = op_shape(ta, m, k)
    Br, Bc = op_shape(tb, k, n)
    A = make_mat(13 + s, Ar, Ac, Ar + pad, "wide", 10, cplx=True)
    B = make_mat(15 + s, Br, Bc, Br + pad, "wide", 10, cplx=True)
    C0 = make_mat(17 + s, m, n, m, "u", cplx=True)
    dC = to_dev(C0)
    oz.zgemm(ta, tb, m, n, k, 1.0 + 0.5j, shifted(A, off), A.shape[0], shifted(B, off), B.shape[0], 0.25 - 1.0j, dC, m, s)
    torch.cuda.synchronize()
    want = C0.copy(order="F")
    assert oracle.zgemm(ta, tb, m, n, k, 1.0 + 0.5j, A, A.shape[0], B, B.shape[0], 0.25 - 1.0j, want, m, s) == 0
    assert np.array_equal(bits(from_dev(dC, C0)), bits(want))


@pytest.mark.parametrize("ops", ["NN", "TT"])
@pytest.mark.parametrize("case", [(20, 18, 140, 16, -1045, 1000), (20, 18, 140, 22, -1045, 1000), (5, 6, 1, 3, 1023, -1060)])
def test_rows_scaled_in_two_factors_and_non_finite_rows(oracle, oz, case, ops):
    """exponents past +-1000, zero rows, and a row with an infinity and one with a NaN"""
    import torch
    m, n, k, s, ea, eb = case
    ta, tb = ops
    Ar, Ac = op_shape(ta, m, k)
    Br, Bc = op_shape(tb, k, n)
    A = np.ldexp(make_mat(23, Ar, Ac, Ar, "u"), ea)
    B = np.ldexp(make_mat(25, Br, Bc, Br, "u"), eb)
    opA = A if ta == "N" else A.T
    opA[2, :] = 0.0
    opA[3, 0] = np.inf
    opA[4, -1] = np.nan
    A, B = np.asfortranarray(A), np.asfortranarray(B)
    C0 = np.zeros((m, n), order="F")
    dC = to_dev(C0)
    oz.gemm(ta, tb, m, n, k, 1.0, to_dev(A), Ar, to_dev(B), Br, 0.0, dC, m, s)
    torch.cuda.synchronize()
    want = C0.copy(order="F")
    assert oracle.dgemm(ta, tb, m, n, k, 1.0, A, Ar, B, Br, 0.0, want, m, s) == 0
    got = from_dev(dC, C0)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(bits(got[ok]), bits(want[ok]))
