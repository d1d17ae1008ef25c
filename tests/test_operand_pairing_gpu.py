"""GPU tests of default-mode results when large entries of one operand meet
small ones of the other (columns of A in mixed units, rows of B in the inverse
units; blocks of rows and columns that are large at different k): they keep
the componentwise bound of a plain product, whichever path serves the call."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

T = {"d": torch.float64, "s": torch.float32, "z": torch.complex128, "c": torch.complex64}
U = {"d": 2.0 ** -53, "z": 2.0 ** -52, "s": 2.0 ** -24, "c": 2.0 ** -23}  # complex products: twice the unit


def scales(kind, k):
    i = torch.arange(k, device="cuda", dtype=torch.float64)
    if kind == "half1e6":
        return torch.where(i % 2 == 0, 1e6, 1.0)
    if kind == "decades":
        return 10.0 ** (i * 10 / k).floor()
    return torch.where(i < k // 2, 2.0 ** 30, 1.0)


def operands(dt, m, n, k, kind, seed=3):
    """op(A) m x k and op(B) k x n as (cols, rows) tensors, C n x m."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def one(rows, cols):
        return (torch.rand((cols, rows), dtype=T[dt], device="cuda", generator=gen) - (0.5 + 0.5j if dt in "zc" else 0.5))

    A, B, C = one(m, k), one(k, n), one(m, n)
    if kind == "blocks":  # rows of A, columns of B: the first half large at even k, the others at odd k
        even = torch.arange(k, device="cuda") % 2 == 0
        first = torch.arange(m, device="cuda") < m // 2
        A = A * torch.where(even[:, None] == first[None, :], 1e8, 1.0).to(T[dt])
        first = torch.arange(n, device="cuda") < n // 2
        B = B * torch.where(even[None, :] == first[:, None], 1e8, 1.0).to(T[dt])
    elif kind != "even":
        s = scales(kind, k)
        A = A * s[:, None].to(T[dt])
        B = B / s[None, :].to(T[dt])
    return A, B, C


def check(out, A, B, C, alpha, beta, k, dt):
    wide = torch.complex128 if dt in "zc" else torch.float64
    A, B, C = A.to(wide), B.to(wide), C.to(wide)
    ref = alpha * (B @ A) + beta * C
    bound = (k + 2) * U[dt] * (abs(alpha) * (B.abs() @ A.abs()) + abs(beta) * C.abs())
    error = (out.to(wide) - ref).abs()
    assert bool((error <= bound).all()), (error / bound).nan_to_num().max().item()


# either side of 6e9 (FP64) and 2e9 (complex128) multiply-adds
SIZES = [("d", (1300, 1301, 1302)), ("d", (2048, 1900, 2000)), ("z", (900, 901, 903)), ("z", (1300, 1280, 1290)),
         ("s", (768, 700, 1024)), ("c", (640, 700, 600))]


@pytest.mark.parametrize("kind", ["half1e6", "decades", "half2^30", "blocks"])
@pytest.mark.parametrize("dt,shape", SIZES)
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T"), ("T", "N")])
def test_unmatched_scales_keep_the_bound(blx, dt, shape, kind, ta, tb):
    m, n, k = shape
    A, B, C = operands(dt, m, n, k, kind)
    out = C.clone()
    a, lda = (A, m) if ta == "N" else (A.mT.contiguous(), k)
    b, ldb = (B, k) if tb == "N" else (B.mT.contiguous(), n)
    rc = blx.gemm_device(ta, tb, m, n, k, 1.5, a, lda, b, ldb, -0.5, out, m, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    check(out, A, B, C, 1.5, -0.5, k, dt)


@pytest.mark.parametrize("dt,shape", [("d", (2100, 1900, 512)), ("s", (1024, 1024, 300))])
def test_few_entries_that_meet_keep_the_bound(blx, dt, shape):
    # one entry in ten: a row and a column share a few dozen products or fewer
    m, n, k = shape
    A, B, C = operands(dt, m, n, k, "even")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    A, B = (x * (torch.rand(x.shape, device="cuda", generator=gen) < 0.1) for x in (A, B))
    out = C.clone()
    rc = blx.gemm_device("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, out, m, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    check(out, A, B, C, 1.0, 0.0, k, dt)


@pytest.mark.parametrize("dt,shape", [("d", (1300, 1300, 1300)), ("d", (2100, 1900, 1600)), ("z", (900, 900, 900))])
def test_decaying_kernels_keep_the_bound(blx, dt, shape):
    # entries that fall off from the diagonal: far from C's diagonal every product is tiny
    m, n, k = shape
    at = [torch.arange(x, device="cuda", dtype=torch.float64) / x for x in (m, n, k)]
    A = torch.exp(-((at[2][:, None] - at[0][None, :]) / 0.1) ** 2).to(T[dt])
    B = torch.exp(-((at[2][None, :] - at[1][:, None]) / 0.1) ** 2).to(T[dt])
    C = torch.zeros((n, m), dtype=T[dt], device="cuda")
    out = C.clone()
    rc = blx.gemm_device("N", "N", m, n, k, 1.0, A.contiguous(), m, B.contiguous(), k, 0.0, out, m, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    check(out, A, B, C, 1.0, 0.0, k, dt)


@pytest.mark.parametrize("dt,shape", SIZES)
def test_matched_scales_stay_emulated(blx, dt, shape):
    # large meets large: nothing is lost, and the call keeps its path
    m, n, k = shape
    A, B, C = operands(dt, m, n, k, "even")
    s = scales("half1e6", k).to(T[dt])
    A, B = A * s[:, None], B * s[None, :]
    out = C.clone()
    rc = blx.gemm_device("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, out, m, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    assert blx.call_stats()["path"] == 2
    check(out, A, B, C, 1.0, 0.0, k, dt)


def test_zero_blocks_stay_emulated(blx):
    # block-diagonal operands: the zero blocks of C are exact and do not count
    m = n = k = 1400
    A, B, C = operands("d", m, n, k, "even")
    half = torch.arange(k, device="cuda") < k // 2
    keep = (half[:, None] == half[None, :]).to(torch.float64)
    A, B = A * keep, B * keep
    out = C.clone()
    rc = blx.gemm_device("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, out, m, dtype="d")
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    assert blx.call_stats()["path"] == 2
    check(out, A, B, C, 1.0, 0.0, k, "d")
    assert not out[:, :m // 2][n // 2:].any()


@pytest.mark.parametrize("uplo", ["U", "L"])
def test_pairs_outside_the_triangle_do_not_count(blx, uplo):
    # SYRK with mixed units: both sides carry the same scale
    n, k = 1700, 1500
    A, _, _ = operands("d", n, n, k, "even")
    A = A * scales("half1e6", k)[:, None]
    C = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    rc = blx.dsyrk_device(uplo, "N", n, k, 1.0, A, n, 0.0, C, n)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    assert blx.call_stats()["path"] == 2
    ref, bound = A.mT @ A, (k + 2) * U["d"] * (A.abs().mT @ A.abs())
    tri = torch.tril if uplo == "L" else torch.triu
    assert bool((tri((C.mT - ref).abs()) <= tri(bound)).all())


@pytest.mark.parametrize("kind", ["half1e6", "decades"])
def test_solve_with_mixed_units(blx, kind):
    # a triangle whose columns are in mixed units: the solution's rows come in the inverse units
    m, n = 2600, 1300
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    A = (torch.rand((m, m), dtype=torch.float64, device="cuda", generator=gen) - 0.5) / m  # (cols, rows)
    A = torch.triu(A) + 2 * torch.eye(m, dtype=torch.float64, device="cuda")               # lower triangle
    A = A * scales(kind, m)[:, None]
    B = torch.rand((n, m), dtype=torch.float64, device="cuda", generator=gen) - 0.5
    X = B.clone()
    rc = blx.dtrsm_device("L", "L", "N", "N", m, n, 1.0, A, m, X, m)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    # backward error of substitution: |A X - B| <= (m + 2) u |A||X|
    ratio = ((X @ A - B).abs() / ((m + 2) * U["d"] * (X.abs() @ A.abs()))).max().item()
    assert ratio <= 1.0, ratio


def test_served_call_with_mixed_units(blx):
    m, n, k = 2048, 1900, 2000
    A, B, C = operands("d", m, n, k, "decades")
    hA, hB, hC = (np.asfortranarray(x.cpu().numpy().T) for x in (A, B, C))
    blx.serve_start(0, 0, 2)
    try:
        blx.cblas_dgemm(102, oracle.TRANS_OF["N"], oracle.TRANS_OF["N"], m, n, k, 1.5, hA, m, hB, k, -0.5, hC, m)
        assert blx.last_status() == blx.BLASX_OK, blx.last_error()
    finally:
        blx.serve_stop()
    check(torch.from_numpy(np.ascontiguousarray(hC.T)).cuda(), A, B, C, 1.5, -0.5, k, "d")
