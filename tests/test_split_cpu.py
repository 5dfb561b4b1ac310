"""The split's two-instruction residue and the GEMM epilogue's FP32 residue.

The split's, exhaustively: for every modulus of every set and every byte
dot product it can meet, the FP32 quotient leaves a byte congruent to the value in [-128, 127]."""
import numpy as np
import pytest

from common import oracle


def moduli():
    o = oracle()
    sets = {m for s in range(2, 25) for m in o.plan(s, 4).m[:s]} | {m for s in range(25, 33) for m in o.plan_ext(s, 4).m[:s]}
    return sorted(int(m) for m in sets)


@pytest.mark.parametrize("m", moduli())
def test_symmetric_residue(m):
    # v' = off + sum of at most 16 products of a byte and a weight below m; complex operands add two
    # such values of at most 12 products each
    top = max(m + 16 * 255 * (m - 1), 2 * (m + 12 * 255 * (m - 1)))
    v = np.arange(top + 1, dtype=np.int64)
    km = (2 ** 23 + m - 1) // m * m
    assert km + top < 2 ** 24  # one float binade: the bits of v are 0x4B000000 + (km - 2^23) + v'
    finv = np.float32(1.0) / np.float32(m)
    num, e = int(np.float64(finv) * 2.0 ** 32), 32  # finv = num 2^-32 exactly (1/256 <= finv < 1/64)
    assert num * 2.0 ** -e == float(finv)
    # round to nearest even of (km + v') finv + 1.5 2^23 to an integer (the result's ulp is 1)
    p = (km + v) * num
    assert p.max() < 2 ** 62
    t = p >> e
    rest = p - (t << e)
    half = 1 << (e - 1)
    t = t + ((rest > half) | ((rest == half) & (t % 2 == 1)))  # 1.5 2^23 is even
    q = t - km // m
    r = v - q * m
    byte = ((0x4B000000 + km - 2 ** 23 + v) - (0x4B400000 + t) * m) % 256
    signed = np.where(byte >= 128, byte - 256, byte)
    if m == 256:
        assert np.array_equal(byte, v % 256)
    else:
        assert r.min() >= -128 and r.max() <= 127
        assert np.array_equal(signed, r)
    assert np.all((signed - v) % m == 0)


@pytest.mark.parametrize("m", moduli())
def test_fp32_residue_of_gemm_sums(m):
    """q = rint(fl(c fl(1/m))) in one rounding for every int32 sum of at most 1024 products (512 for m =
    255), |c| <= 2^24 (2^23): c - q m is a byte in [-128, 127]. q does not decrease with c, so the sums on
    both sides of every tie c = (j + 1/2) m and the ends of the range decide."""
    top = 2 ** 23 if m == 255 else 2 ** 24
    if m == 256:
        return  # the residue is the low byte
    j = np.arange(-top // m - 2, top // m + 2, dtype=np.int64)
    c = np.concatenate([(2 * j + 1) * m // 2 + d for d in (-1, 0, 1, 2)] + [np.array([-top, -top + 1, 0, top - 1, top])])
    c = c[np.abs(c) <= top]
    num, e = int(np.float64(np.float32(1.0) / np.float32(m)) * 2.0 ** 32), 32
    p = c * num
    t = p >> e  # round to nearest even: the addend 1.5 2^23 is even, the sum's ulp 1
    rest = p - (t << e)
    t = t + ((rest > (1 << (e - 1))) | ((rest == (1 << (e - 1))) & (t % 2 == 1)))
    r = c - t * m
    assert r.min() >= -128 and r.max() <= 127
