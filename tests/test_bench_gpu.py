"""bench.py's DGEMM leg reports the launches that a call makes, counted by the library, not a formula."""
import importlib
import sys
import types

import pytest

from common import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [400, 600])
def test_launches_per_call(n):
    import torch
    import oz2
    sys.path.insert(0, ROOT)
    bench = importlib.import_module("bench")
    stream = torch.cuda.current_stream()
    out = bench.dgemm_leg(types.SimpleNamespace(size=n, k=0, s=16), oz2, torch, torch.device("cuda", 0), stream, 0)
    oz = oz2.Ozaki2(stream)
    try:
        A = torch.rand(n * n, dtype=torch.float64, device="cuda")
        C = torch.zeros_like(A)
        before = oz.kernel_launches()
        oz.gemm("N", "N", n, n, n, 1.5, A, n, A, n, -0.5, C, n, 16)
        torch.cuda.synchronize()
        assert out["gpu_launches_per_call"] == oz.kernel_launches() - before
    finally:
        oz.close()
