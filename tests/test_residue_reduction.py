"""CPU restatement of the residue GEMM's reduction of an int32 accumulator
modulo each modulus (one byte dot product and one multiply-high)."""
import random

import pytest

MODULI = (256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181, 179, 173)


def residue_of(x, m):
    biased = (x & 0xFFFFFFFF) ^ 0x80000000
    s = sum(((biased >> (8 * k)) & 255) * (2 ** (8 * k) % m) for k in range(4)) + (m - 2 ** 31 % m) % m
    assert s < 2 ** 20
    return s - (s * -(-2 ** 32 // m) >> 32) * m


@pytest.mark.parametrize("m", MODULI)
def test_reduction_is_the_residue(m):
    rng = random.Random(m)
    edges = [0, 1, -1, m, -m, m - 1, 1 - m, 2 ** 31 - 1, -2 ** 31, 2 ** 30, -2 ** 30, 65536 * 128 * 128]
    for x in edges + [rng.randrange(-2 ** 31, 2 ** 31) for _ in range(2000)]:
        x = (x + 2 ** 31) % 2 ** 32 - 2 ** 31
        assert residue_of(x, m) == x % m
