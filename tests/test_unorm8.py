"""The shading kernels turn a texel byte i into i / 255.0 with one fused
operation on x = i / 256: the result must be the correctly rounded quotient
for every byte."""
from fractions import Fraction

import numpy as np


def round_f32(x):
    """Nearest float32 of a positive Fraction in the normal range, ties to even."""
    e = 0
    while x >= 2:
        x, e = x / 2, e + 1
    while x < 1:
        x, e = x * 2, e - 1
    m = x * 2**23
    n = int(m)
    d = m - n
    n += 1 if d > Fraction(1, 2) or (d == Fraction(1, 2) and n & 1) else 0
    return np.float32(n * 2.0 ** (e - 23))


def test_fused_unorm8_is_the_quotient():
    c = Fraction(float(np.float32(1.0) / np.float32(255.0)))
    for i in range(1, 256):
        x = np.uint32(0x3F800000 | (i << 15)).view(np.float32) - np.float32(1.0)
        assert x == np.float32(i / 256.0)
        xf = Fraction(float(x))
        assert round_f32(xf * c + xf) == np.float32(i) / np.float32(255.0), i
