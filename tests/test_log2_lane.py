"""The table logarithm of the AL16 codes (log2_lane in fullrank_fast.cuh), restated with the same operations on the host."""
import os
import re
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "adafactor-8bit_b200", "csrc")
getcontext().prec = 60


def table():
    with open(os.path.join(CSRC, "log2_lane_table.inc")) as f:
        rows = re.findall(r"\{ 0x([0-9a-f]{8})u, (\S+) \}", f.read())
    return [(Fraction(float(np.array([int(h, 16) << 32], dtype=np.uint64).view(np.float64)[0])), float.fromhex(t)) for h, t in rows]


def coefficients():
    with open(os.path.join(CSRC, "fullrank_fast.cuh")) as f:
        body = f.read().split("float log2_lane(")[1].split("return")[0]
    return [float.fromhex(x) for x in re.findall(r"(-?0x1\.[0-9a-f]+p[+-]\d+)[;)]", body)]


def log2_lane(x, inv_tab, coef):
    b = int(np.float32(x).view(np.uint32))
    near = b + 0x20000
    inv, tab = inv_tab[(near >> 18) & 31]
    e = (near >> 23) - 127
    r = Fraction(float(np.float32(x))) / Fraction(2) ** e * inv - 1
    assert float(r) == r                                     # exact in binary64
    p = coef[0]
    for c in coef[1:]:
        p = float(Fraction(p) * r + Fraction(c))             # fma
    return np.float32(float(Fraction(p) * r + Fraction(float(e + tab))))


@pytest.mark.parametrize("low,high", [(-1e-4, 1e-4), (-0.02, 0.02), (-126.0, 127.9)])
def test_log2_lane_is_correctly_rounded(low, high):
    """Around 1 too, where the result is small: log2 of the sixty-digit decimal, rounded once."""
    inv_tab, coef = table(), coefficients()
    assert len(inv_tab) == 32 and inv_tab[0] == (1, 0.0) and len(coef) == 9
    rng = np.random.default_rng(5)
    for x in (2.0 ** rng.uniform(low, high, 400)).astype(np.float32):
        want = np.float32(float(Decimal(float(x)).ln() / Decimal(2).ln()))
        assert log2_lane(x, inv_tab, coef) == want, float(x)
