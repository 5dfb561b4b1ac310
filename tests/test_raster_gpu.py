"""Raster groups wider than the problem, up to the largest the call takes (the product group_j x tiles would pass 32
bits): the same jobs as one group of all columns, bit for bit against the oracle."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("group_j", [3, 4, 1 << 29, 1 << 30, (1 << 31) - 1])
def test_wide_raster(oracle, oz, bn, group_j):
    import torch
    m, n, k, s = 4 * bn - 1, 260, 40, 14  # four by three tiles
    A, B, C = make_mat(1, m, k, m, "u"), make_mat(2, k, n, k, "u"), np.zeros((m, n), order="F")
    dC = to_dev(C)
    oz.set_gemm_config(bn, group_j, 0)
    try:
        oz.gemm("N", "N", m, n, k, 1.0, to_dev(A), m, to_dev(B), k, 0.0, dC, m, s)
        torch.cuda.synchronize()
        assert oz.gemm_config()["group_j"] == group_j
    finally:
        oz.set_gemm_config(0, 16, 0)
    oz.check_device_error()
    want = C.copy(order="F")
    assert oracle.dgemm("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, want, m, s) == 0
    assert np.array_equal(bits(from_dev(dC, C)), bits(want))
