"""The GEMM's FP32 residues (few k-blocks) on both sides of their limits, bit for bit against the oracle:
4 k-blocks (k = 512) for sets with m = 255, 8 (k = 1024) for the others, with largest-magnitude data
(residue sums near their bound), and a grouped call that mixes both kinds."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["u", "maxmag"])
@pytest.mark.parametrize("k", [1, 128, 512, 513, 1024, 1025])
@pytest.mark.parametrize("s", [4, 6, 13, 16, 22])
def test_dgemm(oracle, oz, s, k, kind):
    import torch
    m, n = 133, 70
    A, B = make_mat(s, m, k, m, kind), make_mat(s + 1, k, n, k, kind)
    C0 = make_mat(3, m, n, m, "u")
    dC = to_dev(C0)
    oz.gemm("N", "N", m, n, k, 1.5, to_dev(A), m, to_dev(B), k, -0.5, dC, m, s)
    torch.cuda.synchronize()
    want = C0.copy(order="F")
    assert oracle.dgemm("N", "N", m, n, k, 1.5, A, m, B, k, -0.5, want, m, s) == 0
    assert np.array_equal(bits(from_dev(dC, C0)), bits(want))


def test_grouped_mix(oracle, oz):
    import torch
    specs = [(40, 300, 100, 14), (300, 60, 1100, 14), (129, 129, 900, 6), (33, 257, 600, 17), (64, 64, 2000, 17)]
    probs, keep = [], []
    for i, (m, n, k, s) in enumerate(specs):
        A, B, C = make_mat(i, m, k, m, "u"), make_mat(9 + i, k, n, k, "u"), np.zeros((m, n), order="F")
        dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
        probs.append(("N", "N", m, n, k, 1.0, dA, m, dB, k, 0.0, dC, m, s))
        keep.append((A, B, C, dC))
    oz.gemm_grouped(probs)
    torch.cuda.synchronize()
    for (m, n, k, s), (A, B, C, dC) in zip(specs, keep):
        want = C.copy(order="F")
        assert oracle.dgemm("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, want, m, s) == 0
        assert np.array_equal(bits(from_dev(dC, C)), bits(want)), (m, n, k, s)
