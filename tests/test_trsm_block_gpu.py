"""GPU tests of the substitution kernel at the edges of its blocks (256 rows),
row groups (32) and panels (16): backward error of the solve, with NaN in the
triangle (and the unit diagonal) that must not be read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}
ORDERS = [1, 15, 17, 32, 33, 255, 256, 257, 300]


@pytest.mark.parametrize("dt", "sdcz")
@pytest.mark.parametrize("side,nvec", [("L", 1), ("L", 37), ("R", 3), ("R", 65)])
@pytest.mark.parametrize("uplo,trans,diag", [("U", "N", "N"), ("L", "N", "U"), ("U", "C", "N"), ("L", "T", "N")])
@pytest.mark.parametrize("K", ORDERS)
def test_block_edges(blx, dt, side, nvec, uplo, trans, diag, K):
    T = DT[dt]
    rng = np.random.default_rng(K * 7 + nvec)

    def rand(*shape):
        x = rng.uniform(-1, 1, shape)
        return (x + 1j * rng.uniform(-1, 1, shape) if dt in "cz" else x).astype(T)

    A = np.asfortranarray(rand(K, K) / K + 2 * np.eye(K)).astype(T, order="F")
    keep = np.triu(np.ones((K, K), bool)) if uplo == "U" else np.tril(np.ones((K, K), bool))
    if diag == "U":
        keep &= ~np.eye(K, dtype=bool)
    S = np.where(keep, A, 0)
    if diag == "U":
        S = S + np.eye(K)
    A[~keep] = np.nan
    M, N = (K, nvec) if side == "L" else (nvec, K)
    B0 = np.asfortranarray(rand(M, N))
    X = B0.copy(order="F")
    alpha = -0.5
    call = {"s": blx.cblas_strsm, "d": blx.cblas_dtrsm, "c": blx.cblas_ctrsm, "z": blx.cblas_ztrsm}[dt]
    call(blx.CblasColMajor, blx.SIDE[side], blx.UPLO[uplo], blx.TRANS[trans], blx.DIAG[diag], M, N, alpha, A, K, X, M)
    assert blx.last_status() == blx.BLASX_OK, blx.last_error()
    wide = np.clongdouble if dt in "cz" else np.longdouble
    Sw = {"N": S, "T": S.T, "C": S.conj().T}[trans].astype(wide)
    Xw, Bw = X.astype(wide), alpha * B0.astype(wide)
    R = (Sw @ Xw if side == "L" else Xw @ Sw) - Bw
    aS, aX = np.abs(Sw), np.abs(Xw)
    # K + 2 roundings per entry on both sides of the residual; complex products count double
    u = np.finfo(T).eps / 2 * (2 if dt in "cz" else 1)
    bound = 2 * (K + 2) * u * ((aS @ aX if side == "L" else aX @ aS) + np.abs(Bw))
    assert (np.abs(R) <= bound).all()
