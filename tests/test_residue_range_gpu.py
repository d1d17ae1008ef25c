"""GPU tests of the device's residues at the ends of their ranges, against exact
integers: scaled integers of every magnitude below 2^62 for all 20 moduli, and
INT32 accumulators of the residue GEMM near 2^30."""
import random

import numpy as np
import pytest
import torch

from oracle import ozaki_ref

pytestmark = pytest.mark.gpu


@pytest.fixture
def emulated(blx):
    prev = blx.set_dgemm_mode(blx.MODE_OZAKI)
    yield blx
    blx.set_dgemm_mode(prev)


def product(blx, A, B, ta, tb):
    """op(A) B for A (m x k) and B (k x n), stored transposed as ta, tb say; the modulus count."""
    m, k = A.shape
    n = B.shape[1]
    dA = torch.from_numpy(np.ascontiguousarray(A.T if ta == "N" else A)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B.T if tb == "N" else B)).cuda()
    dC = torch.zeros((n, m), dtype=torch.float64, device="cuda")
    rc = blx.gemm_device(ta, tb, m, n, k, 1.0, dA, m if ta == "N" else k, dB, k if tb == "N" else n, 0.0, dC, m)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    st = blx.call_stats()
    assert st["path"] == 2
    return dC.cpu().numpy().T, st["moduli"]


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
def test_every_magnitude_with_all_moduli(emulated, ta, tb):
    # rows [2^61, x, 0, ...]: scaled by one, so x itself is reduced; columns
    # [0, y, 0, ...]: scaled into [2^61, 2^62). So few entries in a long row
    # take every modulus. Products of two doubles, correctly rounded.
    rng = random.Random(2)
    k = 4096
    xs = [s * (2 ** b - 1) for b in range(1, 54) for s in (1, -1)] + [2.0 ** b for b in range(62)]
    xs += [float(rng.randrange(2 ** 53)) * 2.0 ** rng.randrange(-3, 9) // 1 for _ in range(150)]
    xs = [float(x) for x in xs if abs(x) < 2 ** 61]
    xs += [s * float(2 ** 62 - 2 ** 9) for s in (1, -1)]  # the largest: the row's own maximum
    ys = [1.0, -1.0, float(2 ** 53 - 1), -float(2 ** 53 - 1), 3.0, 2.0 / 3.0] + [rng.uniform(-1, 1) for _ in range(60)]
    A, B = np.zeros((len(xs), k)), np.zeros((k, len(ys)))
    A[:, 0], A[:, 1], B[1] = 2.0 ** 61, xs, ys
    C, moduli = product(emulated, A, B, ta, tb)
    assert moduli == ozaki_ref.MODULI.__len__()
    np.testing.assert_array_equal(C, np.array(xs)[:, None] * np.array(ys)[None, :])


def test_accumulators_near_their_bound(emulated):
    # 65536 equal entries v in [2^48, 2^49): scaled by one under 15 moduli.
    # For each of those one row and one column are at the end of the residue's
    # range, so their accumulators reach 65536 h^2
    k, n = 65536, 15
    Q = ozaki_ref.crt(n)[3]
    assert Q == 57
    vs = []
    for m in ozaki_ref.MODULI[:n]:
        h = 127 if m == 256 else (m - 1) // 2
        base = 2 ** 48 + 2 ** 47 + (-(2 ** 48 + 2 ** 47)) % m  # a multiple of m
        vs += [base + h, base - h]
    A = np.repeat(np.array(vs, dtype=np.float64)[:, None], k, axis=1)
    C, moduli = product(emulated, A, A.T.copy(), "T", "N")
    assert moduli == n
    want = np.array([[float(k * p * q) for q in vs] for p in vs])
    np.testing.assert_array_equal(C, want)
