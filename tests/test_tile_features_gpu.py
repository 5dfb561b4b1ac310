"""The fused scale + statistics pass and the features at the edges of its blocks (32 and 8 rows, 8 and 32
inner indices, unrolled by 8, up to its largest k), with zeros, subnormals and both layouts in one call, against
the numpy restatement: every feature but the logarithm exactly."""
import numpy as np
import pytest

import adaptive_oracle
from common import op_shape, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 9, 7), (33, 8, 9), (32, 7, 33), (64, 65, 255), (513, 33, 513),
                                   (40, 512, 2049), (9, 33, 16384)])
def test_edges(oracle, m, n, k):
    import torch
    import oz2
    rng = np.random.default_rng(m * 1000 + k)
    probs, dev = [], []
    for ta, tb in ("NN", "NT", "TN", "TT"):
        Ar, Ac = op_shape(ta, m, k)
        Br, Bc = op_shape(tb, k, n)

        def values(r, c):
            X = (rng.random((r, c)) - 0.5) * np.exp(5.0 * rng.standard_normal((r, c)))
            X[rng.random(X.shape) < 0.1] = 0.0
            X[rng.random(X.shape) < 0.02] = 3e-310
            X[r // 2, :] = 0.0
            return np.asfortranarray(X)

        A, B = values(Ar, Ac), values(Br, Bc)
        probs.append((ta, tb, m, n, k, A, B))
        dev.append((ta, tb, m, n, k, 1.0, to_dev(A), Ar, to_dev(B), Br, 0.0,
                    torch.zeros(m * n, dtype=torch.float64, device="cuda"), m, 16))
    h = oz2.Ozaki2(torch.cuda.current_stream())
    try:
        h.set_adaptive_options(512, 0.9)
        feat, s_an = h.tile_features(dev)
        got, got_s = feat.cpu().numpy(), s_an.cpu().numpy()
    finally:
        h.close()
    want, want_s = adaptive_oracle.tile_features(oracle, probs)
    assert got.shape == want.shape
    np.testing.assert_allclose(got[:, 0], want[:, 0], rtol=1e-6)
    assert np.array_equal(got[:, 1:], want[:, 1:])
    assert np.array_equal(got_s, want_s)
