"""The two-operation quotients by cs^2 and cs^4 (lattice.cuh, over_cs2 ...)
round like the division they replace: x h + RN(x l), the sum rounded once,
with h = RN(1/c) and l = RN(1/c - h).

The computed sum is within 2^-105 (relative) of x / c before its last
rounding, and a quotient of two binary64 numbers that is no midpoint is at
least 2^-107 away from one for every unit of delta = X 2^(k+1) - (2 M + 1) C
(X, C the significands, M the quotient's): only |delta| <= 4 can go wrong, and
each delta has one X per residue of C, so those X are all tried (to 64).  In
binary32 every significand is tried.  Exact rational arithmetic throughout."""
from fractions import Fraction as F
import math
import os
import re

import numpy as np
import pytest

LATTICE = os.path.join(os.path.dirname(__file__), "..", "cfd_cavity_b200", "csrc", "lattice.cuh")


def constants(kind):
    """I2H, I2L, I4H, I4L of CsInv<kind> as the source has them."""
    with open(LATTICE) as fh:
        body = re.search(r"struct CsInv<%s> \{(.*?)\};" % kind, fh.read(), re.S).group(1)
    val = {}
    for name, text in re.findall(r"(I\dH|I\dL) = ([^,;]+)", body):
        text = text.strip().rstrip("f") if "0x" not in text else text.strip()
        val[name] = float.fromhex(text.rstrip("f")) if "0x" in text and "p" in text else float(text)
    return val


def to_double(q):
    return q.numerator / q.denominator  # int / int rounds correctly


@pytest.mark.parametrize("which", ["2", "4"])
def test_binary64_hard_cases(which):
    c = 1.0 / 3.0 if which == "2" else (1.0 / 3.0) * (1.0 / 3.0)
    k = constants("double")
    h, lo = k["I%sH" % which], k["I%sL" % which]
    assert h == to_double(1 / F(c)) and lo == to_double(1 / F(c) - F(h))

    def quotient(x):
        return to_double(x * F(h) + F(to_double(x * F(lo))))

    C = int(math.frexp(c)[0] * 2**53)
    odd = C
    while odd % 2 == 0:
        odd //= 2
    tried = 0
    for shift in (52, 53):
        inv = pow(2, -(shift + 1), odd)
        for delta in range(-64, 65):
            x = delta * inv % odd
            while x < 2**53:
                if x >= 2**52:
                    tried += 1
                    assert quotient(F(x)) == to_double(F(x) / F(c)), (x, delta)
                x += odd
    assert tried > 100
    rng = np.random.default_rng(5)
    for x in rng.integers(2**52, 2**53, 4000):
        assert quotient(F(int(x))) == to_double(F(int(x)) / F(c))


@pytest.mark.parametrize("which", ["2", "4"])
def test_binary32_every_significand(which):
    third = np.float32(1.0) / np.float32(3.0)
    c = third if which == "2" else third * third
    k = constants("float")
    h, lo = k["I%sH" % which], k["I%sL" % which]
    assert h == np.float32(h) and lo == np.float32(lo)
    x = np.arange(2**23, 2**24, dtype=np.float32)
    t = x * np.float32(lo)
    # x h + t fits binary64 exactly (at most 51 bits), so this rounds once
    s = (x.astype(np.float64) * h + t.astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(s, x / c)
