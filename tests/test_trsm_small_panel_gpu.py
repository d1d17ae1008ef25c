"""GPU tests of the complex128 triangular solve with more right-hand sides than
one CTA per SM takes (panels of 8 columns in the substitution kernel): block
sizes on either side of a panel, every form of op(A), both sides."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,uplo", [("L", "U"), ("L", "L"), ("R", "U"), ("R", "L")])
@pytest.mark.parametrize("trans", ["N", "T", "C"])
@pytest.mark.parametrize("order,diag", [(1, "N"), (7, "U"), (8, "N"), (9, "N"), (31, "N"), (33, "U"), (250, "N"), (256, "N"),
                                        (265, "N")])
def test_backward_error(blx, side, uplo, trans, diag, order):
    vecs = 1193  # 150 CTAs of 8 vectors, the last one not full
    m, n = (order, vecs) if side == "L" else (vecs, order)
    rng = np.random.default_rng(order)

    def entries(r, c):
        return np.asfortranarray((rng.random((r, c)) - 0.5) + 1j * (rng.random((r, c)) - 0.5))

    A, B = entries(order, order) / order, entries(m, n)
    A[np.diag_indices(order)] += 2
    X = B.copy(order="F")
    blx.cblas_ztrsm(102, blx.SIDE[side], blx.UPLO[uplo], oracle.TRANS_OF[trans], blx.DIAG[diag], m, n, 1.5, A, order, X, m)
    assert blx.last_status() == blx.BLASX_OK, blx.last_error()
    T = np.triu(A) if uplo == "U" else np.tril(A)
    if diag == "U":
        T = T - np.diag(np.diag(T)) + np.eye(order)
    op = {"N": T, "T": T.T, "C": T.conj().T}[trans]
    op, X, B = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (op, X, B))
    res, mag = (op @ X, op.abs() @ X.abs()) if side == "L" else (X @ op, X.abs() @ op.abs())
    # |op(A) X - alpha B| <= (order + 2) u (|op(A)||X| + |alpha B|), complex products twice the unit
    bound = (order + 2) * 2.0 ** -52 * (mag + 1.5 * B.abs())
    assert bool(((res - 1.5 * B).abs() <= bound).all())
