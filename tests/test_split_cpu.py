"""The split's two-instruction residue, exhaustively: for every modulus of every set and every byte
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
