"""CPU restatement of the slicing's FP32 residue reduction, for every modulus
that uses it: congruent, at most 127 in magnitude, exact in FP32."""
import random
from fractions import Fraction

import numpy as np
import pytest

MODULI = (253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181, 179, 173)


def residue(v, m):
    biased = v + 2 ** 62
    s = sum(((biased >> (8 * k)) & 255) * (2 ** (8 * k) % m) for k in range(8)) + -2 ** 62 % m
    base = 256 * m * -(-12582912 // (256 * m))
    F = base + s
    assert 2 ** 23 <= F < 2 ** 24  # an exact float whose unit is one
    t = round(Fraction(float(np.float32(1.0) / np.float32(m))) * F + 12582912)  # one FMA: half to even
    q = t - (12582912 + base // m)
    assert 2 ** 23 <= t < 2 ** 24 and 12582912 + base // m < 2 ** 24 and abs(q) < 2 ** 24
    out = F - q * m
    assert 2 ** 23 <= out < 2 ** 24
    r = out & 255
    return r - 256 if r >= 128 else r


@pytest.mark.parametrize("m", MODULI)
def test_residue_is_congruent_and_fits(m):
    rng = random.Random(m)
    edges = [0, 1, -1, 2 ** 62 - 1, 1 - 2 ** 62, m // 2, -(m // 2), m // 2 + 1, 2 ** 61 + m // 2]
    for v in edges + [rng.randrange(1 - 2 ** 62, 2 ** 62) >> rng.randrange(62) for _ in range(3000)]:
        r = residue(v, m)
        assert (r - v) % m == 0 and abs(r) <= 127
