"""ZGEMM on both sides of the rule that takes the scale pass into the first launch (complex: k up to 256), every op letter,
padded leading dimensions, a zero row and a zero column, bit for bit against the oracle."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["NN", "CT", "TC"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 31, 255), (31, 33, 256), (40, 65, 257)])
def test_edges(oracle, oz, m, n, k, op):
    import torch
    sa, sb = ((m, k) if op[0] == "N" else (k, m)), ((k, n) if op[1] == "N" else (n, k))
    la, lb = sa[0] + 3, sb[0] + 1
    A, B = make_mat(m, sa[0], sa[1], la, "u", cplx=True), make_mat(n, sb[0], sb[1], lb, "u", cplx=True)
    A[sa[0] // 2, :] = 0.0
    B[:, sb[1] // 2] = 0.0
    C = make_mat(5, m, n, m, "u", cplx=True)
    dC = to_dev(C)
    oz.zgemm(op[0], op[1], m, n, k, 1.5 - 0.5j, to_dev(A), la, to_dev(B), lb, 0.25 + 1.0j, dC, m, 15)
    torch.cuda.synchronize()
    oz.check_device_error()
    want = C.copy(order="F")
    assert oracle.zgemm(op[0], op[1], m, n, k, 1.5 - 0.5j, A, la, B, lb, 0.25 + 1.0j, want, m, 15) == 0
    assert np.array_equal(bits(from_dev(dC, C)), bits(want))
