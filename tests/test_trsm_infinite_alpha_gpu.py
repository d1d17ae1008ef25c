"""GPU test of an infinite alpha in a triangular solve: only the rows of B are
scaled by it, not the rows that pad a block of the substitution kernel."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,uplo,trans", [("L", "U", "N"), ("L", "L", "T"), ("L", "L", "N"), ("R", "L", "N"), ("R", "U", "T"),
                                             ("R", "U", "N")])
@pytest.mark.parametrize("diag", ["N", "U"])
@pytest.mark.parametrize("order", [1, 20, 33, 250, 256, 300])
def test_infinite_alpha(blx, side, uplo, trans, diag, order):
    # positive right-hand sides, a positive diagonal and negative entries
    # beside it: every term of every solution is +inf, in both directions
    m, n = (order, 7) if side == "L" else (7, order)
    A = -torch.ones((order, order), dtype=torch.float64, device="cuda") + 3 * torch.eye(order, dtype=torch.float64, device="cuda")
    B = torch.ones((n, m), dtype=torch.float64, device="cuda")
    rc = blx.dtrsm_device(side, uplo, trans, diag, m, n, float("inf"), A, order, B, m)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    assert bool((B == float("inf")).all())


@pytest.mark.parametrize("order", [20, 250])
def test_infinite_alpha_single(blx, order):
    A = np.asfortranarray(-np.ones((order, order), np.float32) + 3 * np.eye(order, dtype=np.float32))
    B = np.ones((order, 5), np.float32, order="F")
    blx.cblas_strsm(102, blx.SIDE["L"], blx.UPLO["U"], oracle.TRANS_OF["N"], blx.DIAG["N"], order, 5, float("inf"), A, order, B, order)
    assert blx.last_status() == blx.BLASX_OK, blx.last_error()
    assert np.isposinf(B).all()
