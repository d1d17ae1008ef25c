"""GPU tests of the native FP64 / complex128 kernel's tile geometries and of
the k extent cut over a cluster, at tile edges and remainders.

Integer-valued operands of at most 2^20 in magnitude whose products and sums
stay below 2^53 make every order of summation exact, so the comparison is for
equality.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): one 32x32 tile and its edges with k cuts of 1 to 16; 64x48 and 64x64 grids; remainders in every direction
SHAPES = [(1, 1, 1), (31, 33, 65), (32, 32, 512), (33, 31, 1000), (96, 64, 5000), (65, 47, 33), (400, 300, 250),
          (1003, 777, 100), (1500, 900, 64), (2100, 1900, 40)]


@pytest.fixture
def native(blx):
    prev = blx.set_dgemm_mode(blx.MODE_NATIVE)
    yield blx
    blx.set_dgemm_mode(prev)


def stored(rng, rows, cols, dt, pad):
    x = rng.integers(-1000, 1001, (cols, rows + pad)).astype(np.float64)
    if dt == "z":
        x = x + 1j * rng.integers(-1000, 1001, x.shape)
    return x


@pytest.mark.parametrize("dt", ["d", "z"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("C", "C")])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("pad", [0, 1])
def test_tiles_are_exact_on_integers(native, blx, dt, ta, tb, shape, pad):
    M, N, K = shape
    rng = np.random.default_rng(M * 31 + N * 7 + K)
    A = stored(rng, *((M, K) if ta == "N" else (K, M)), dt, pad)
    B = stored(rng, *((K, N) if tb == "N" else (N, K)), dt, pad)
    C = stored(rng, M, N, dt, pad)

    def op(x, rows, t):
        x = x[:, :rows]
        return x.T if t == "N" else (x.conj() if t == "C" else x)

    want = C.copy()
    want[:, :M] = (2 * (op(A, A.shape[1] - pad, ta) @ op(B, B.shape[1] - pad, tb)) - 3 * C[:, :M].T).T
    dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
    rc = blx.gemm_device(ta, tb, M, N, K, 2.0, dA, A.shape[1], dB, B.shape[1], -3.0, dC, M + pad, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    np.testing.assert_array_equal(dC.cpu().numpy(), want)


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n,k", [(33, 1000), (96, 3000), (500, 70), (1300, 40)])
def test_triangular_tiles_are_exact_on_integers(native, blx, uplo, n, k):
    rng = np.random.default_rng(n + k)
    A, C = stored(rng, n, k, "d", 0), stored(rng, n, n, "d", 0)
    full = A.T @ A + 2 * C.T
    keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    want = np.where(keep, full, C.T).T
    dA, dC = torch.from_numpy(A).cuda(), torch.from_numpy(C).cuda()
    assert blx.dsyrk_device(uplo, "N", n, k, 1.0, dA, n, 2.0, dC, n) == blx.BLASX_OK, blx.last_error()
    np.testing.assert_array_equal(dC.cpu().numpy(), want)
