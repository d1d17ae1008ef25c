"""CPU tests of the oracle's restatement of the device's residues: congruent to
the value, within int8, and good for an exact product."""
import random

import numpy as np
import pytest

from oracle import ozaki_ref


@pytest.mark.parametrize("m", ozaki_ref.MODULI)
def test_congruent_and_in_range(m):
    rng = random.Random(m)
    vs = [0, 1, -1, (1 << 62) - 512, 512 - (1 << 62), m // 2, -(m // 2), m // 2 + 1]
    vs += [rng.randrange(1 - (1 << 62), 1 << 62) >> rng.randrange(62) for _ in range(1500)]
    for v in vs:
        r = ozaki_ref.device_residue(v, m)
        assert (r - v) % m == 0 and -128 <= r <= 127 and (m == 256 or abs(r) <= (m + 1) // 2)


def test_products_of_device_residues_reconstruct_exactly():
    rng = random.Random(8)
    for n in (6, 15, 20):
        ms, M, w, Q = ozaki_ref.crt(n)
        top = 1 << min(62, Q - 4)  # 64 entries below 2^(Q - 4): a norm below 2^Q
        a = [rng.randrange(-top, top) for _ in range(64)]
        b = [rng.randrange(-top, top) for _ in range(64)]
        x = 0
        for l, m in enumerate(ms):
            ra, rb = ([ozaki_ref.device_residue(v, m) for v in vs] for vs in (a, b))
            x += sum(p * q for p, q in zip(ra, rb)) % m * w[l]
        x %= M
        assert (x - M if 2 * x >= M else x) == sum(p * q for p, q in zip(a, b))
    assert np.int8(-128) == -128  # the lowest residue (m = 256) is an int8
