"""Launches that share operands of both layouts and start while the one before drains: chains of products that
read the previous result at once, on the default and on a side stream, and grouped calls with every op pair
(descriptors as a kernel parameter and through the staging ring), bit for bit against the oracle."""
import numpy as np
import pytest

from common import bits, from_dev, make_mat, to_dev

pytestmark = pytest.mark.gpu
OPS = ("NN", "NT", "TN", "TT")


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("n,s", [(1, 14), (40, 6), (129, 16), (260, 20)])
def test_chain(oracle, oz, n, s, side):
    import torch
    A, B = make_mat(1, n, n, n, "u"), make_mat(2, n, n, n, "u")
    dA, dB, outs = to_dev(A), to_dev(B), [to_dev(np.zeros((n, n), order="F")) for _ in range(6)]
    torch.cuda.synchronize()
    st = torch.cuda.Stream() if side else None
    if side:
        oz.set_stream(st.cuda_stream)
    try:
        for i, out in enumerate(outs):
            src, op = (outs[i - 1] if i else dA), OPS[i % 4]
            oz.gemm(op[0], op[1], n, n, n, 1.0, src, n, dB, n, 0.0, out, n, s)
        torch.cuda.synchronize()
    finally:
        if side:
            oz.set_stream(0)
    x = A
    for i, out in enumerate(outs):
        want, op = np.zeros((n, n), order="F"), OPS[i % 4]
        assert oracle.dgemm(op[0], op[1], n, n, n, 1.0, x, n, B, n, 0.0, want, n, s) == 0
        assert np.array_equal(bits(from_dev(out, want)), bits(want)), i
        x = want


@pytest.mark.parametrize("copies", [1, 24])
def test_grouped_layouts(oracle, oz, copies):
    import torch
    probs, keep = [], []
    for i in range(8 * copies):
        m, n, k, s, op = 30 + i % 8 * 17, 140 - i % 8 * 13, 1 + i % 8 * 37, (8, 14, 20)[i % 3], OPS[i % 4]
        sa, sb = ((m, k) if op[0] == "N" else (k, m)), ((k, n) if op[1] == "N" else (n, k))
        A, B = make_mat(i, sa[0], sa[1], sa[0], "u"), make_mat(i + 99, sb[0], sb[1], sb[0], "u")
        C = np.zeros((m, n), order="F")
        dC = to_dev(C)
        probs.append((op[0], op[1], m, n, k, 1.0, to_dev(A), sa[0], to_dev(B), sb[0], 0.0, dC, m, s))
        keep.append((A, B, C, dC))
    oz.gemm_grouped(probs)
    torch.cuda.synchronize()
    for p, (A, B, C, dC) in zip(probs, keep):
        want = C.copy(order="F")
        assert oracle.dgemm(p[0], p[1], p[2], p[3], p[4], 1.0, A, p[7], B, p[9], 0.0, want, p[2], p[13]) == 0
        assert np.array_equal(bits(from_dev(dC, C)), bits(want)), p[:5]


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 31), (32, 64, 32), (33, 31, 33), (65, 40, 511), (40, 65, 512),
                                   (33, 33, 513)])
def test_first_launch(oracle, oz, m, n, k, op):
    """the scale pass in the first launch (k up to 512) and beyond it, padded leading dimensions, a zero row"""
    import torch
    sa, sb = ((m, k) if op[0] == "N" else (k, m)), ((k, n) if op[1] == "N" else (n, k))
    la, lb = sa[0] + 3, sb[0] + 1
    A, B = make_mat(m, sa[0], sa[1], la, "u"), make_mat(n, sb[0], sb[1], lb, "u")
    A[sa[0] // 2, :] = 0.0
    C = make_mat(5, m, n, m, "u")
    dC = to_dev(C)
    oz.gemm(op[0], op[1], m, n, k, 1.5, to_dev(A), la, to_dev(B), lb, -0.5, dC, m, 15)
    torch.cuda.synchronize()
    want = C.copy(order="F")
    assert oracle.dgemm(op[0], op[1], m, n, k, 1.5, A, la, B, lb, -0.5, want, m, 15) == 0
    assert np.array_equal(bits(from_dev(dC, C)), bits(want))


@pytest.mark.parametrize("k", [300, 700])
def test_user_capture(oracle, oz, k):
    """a product captured by the caller into a CUDA graph (chained launches become graph edges), replayed on new data"""
    import torch
    m, n, s = 150, 90, 14
    dA, dB, dC = to_dev(np.zeros((m, k), order="F")), to_dev(np.zeros((k, n), order="F")), to_dev(np.zeros((m, n), order="F"))
    st = torch.cuda.Stream()
    oz.set_stream(st.cuda_stream)
    try:
        oz.gemm("N", "N", m, n, k, 1.0, dA, m, dB, k, 0.0, dC, m, s)  # the workspace grows outside the capture
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            oz.gemm("N", "N", m, n, k, 1.0, dA, m, dB, k, 0.0, dC, m, s)
        for seed in (1, 2):
            A, B = make_mat(seed, m, k, m, "u"), make_mat(seed + 7, k, n, k, "u")
            dA.copy_(to_dev(A))
            dB.copy_(to_dev(B))
            g.replay()
            torch.cuda.synchronize()
            want = np.zeros((m, n), order="F")
            assert oracle.dgemm("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, want, m, s) == 0
            assert np.array_equal(bits(from_dev(dC, want)), bits(want))
    finally:
        torch.cuda.synchronize()
        oz.set_stream(0)
