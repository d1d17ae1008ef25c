"""GPU tests of the emulated path's statistics and modulus decision: every
entry of both operands counts, whatever the layout, at the edges of the row
groups (8 or 64 rows) and of the k-chunks."""
import math

import numpy as np
import pytest

import torch

from test_ozaki_gpu import make

pytestmark = pytest.mark.gpu

MODULI = (256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181, 179, 173)
SHAPES = [(1, 65, 129), (65, 9, 5000), (8, 64, 128), (300, 1, 33), (7, 130, 2305)]


def run(blx, dt, ta, tb, M, N, K, A, B, beta, C):
    """The device-resident call on copies of the operands; C is updated, the call statistics come back."""
    dA, dB, dC = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (A, B, C))
    code = {np.float64: "d", np.float32: "s", np.complex128: "z"}[dt]
    rc = blx.gemm_device(ta, tb, M, N, K, 1.0, dA, A.shape[0], dB, B.shape[0], beta, dC, M, dtype=code)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    C[...] = dC.cpu().numpy().T
    return blx.call_stats()


@pytest.fixture
def emulated(blx):
    prev = blx.set_dgemm_mode(blx.MODE_OZAKI)
    yield blx
    blx.set_dgemm_mode(prev)


def expected_moduli(opA, opB, unit):
    """The documented rule, restated: the smallest N with 3 rho_A rho_B 2^-q(N) / u <= 1/2."""
    K = opA.shape[1]
    rho, h = [], []
    for X in (opA, opB.T):
        parts = np.abs(np.stack([X.real, X.imag])) if np.iscomplexobj(X) else np.abs(X)[None]
        parts = parts.astype(np.float64)
        n2, n1, mx = np.sqrt((parts ** 2).sum((0, 2))), parts.sum((0, 2)), parts.max((0, 2))
        rho.append(max(1.0, (n2 * math.sqrt(K) / n1).max()))
        h.append(math.log2((n2 / mx).min()))
    prod, est = 1, None
    for n, m in enumerate(MODULI, 1):
        prod *= m
        Q = math.floor((math.log2(prod) - 2) / 2)
        est = 3 * rho[0] * rho[1] * 2.0 ** -min(min(Q, 62 + h[0]), min(Q, 62 + h[1])) / unit
        if n >= 6 and est <= 0.5:
            assert est < 0.499  # the inputs leave no doubt about the count
            return n
        assert n < 6 or est > 0.501
    return 20


@pytest.mark.parametrize("dt", [np.float64, np.float32, np.complex128])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T"), ("N", "T"), ("T", "N")])
@pytest.mark.parametrize("shape", SHAPES)
def test_modulus_count_follows_the_rule(emulated, blx, dt, ta, tb, shape):
    M, N, K = shape
    A, _, B, _, C = make(dt, ta, tb, M, N, K, 5)
    A[tuple(s - 1 for s in A.shape)] *= 40  # the last entry alone sets the spread
    opA, opB = (A if ta == "N" else A.T), (B if tb == "N" else B.T)
    st = run(blx, dt, ta, tb, M, N, K, A, B, 0.0, C)
    assert st["path"] == 2
    assert st["moduli"] == expected_moduli(opA, opB, 2.0 ** (-24 if dt == np.float32 else -53))


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
@pytest.mark.parametrize("shape", SHAPES)
def test_a_single_nonfinite_entry_is_seen(emulated, blx, ta, tb, shape):
    M, N, K = shape
    A, _, B, _, C0 = make(np.float64, ta, tb, M, N, K, 6)
    for which, (r, c) in [("A", (0, 0)), ("A", (-1, -1)), ("B", (0, -1)), ("B", (-1, 0))]:
        X = {"A": A, "B": B}
        Y = {k: v.copy(order="F") for k, v in X.items()}
        Y[which][r, c] = np.inf
        C = C0.copy(order="F")
        st = run(blx, np.float64, ta, tb, M, N, K, Y["A"], Y["B"], 0.5, C)
        assert st["path"] == 4  # the native kernel, chosen on the device
        want = C0.copy(order="F")
        blx.set_dgemm_mode(blx.MODE_NATIVE)
        run(blx, np.float64, ta, tb, M, N, K, Y["A"], Y["B"], 0.5, want)
        blx.set_dgemm_mode(blx.MODE_OZAKI)
        np.testing.assert_array_equal(C, want)
