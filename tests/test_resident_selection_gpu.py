"""GPU tests of the lower line from which device-resident calls emulate: on
either side of it, for operands of wide spread, and without memory for the
scratch, where the native kernel's result is expected bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

T = {"d": torch.float64, "z": torch.complex128}


def operands(dt, m, n, k, spread=0.0):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n + k)

    def one(rows, cols):
        x = torch.rand((cols, rows), dtype=T[dt], device="cuda", generator=gen) - 0.5
        if spread:
            x = x * torch.exp(spread * torch.randn((cols, rows), dtype=torch.float64, device="cuda", generator=gen))
        return x

    return one(m, k), one(k, n), one(m, n)


def call(blx, dt, m, n, k, A, B, C, mode=0):
    prev = blx.set_dgemm_mode(mode)
    out = C.clone()
    rc = blx.gemm_device("N", "N", m, n, k, 1.5, A, m, B, k, -0.5, out, m, dtype=dt)
    blx.set_dgemm_mode(prev)
    assert rc == blx.BLASX_OK, blx.last_error()
    torch.cuda.synchronize()
    return out, blx.call_stats()["path"]


@pytest.mark.parametrize("dt,below,above", [("d", (1250, 1260, 1250), (1260, 1270, 1260)), ("z", (880, 890, 880), (890, 900, 890))])
def test_the_line(blx, dt, below, above):
    for shape, path in ((below, 1), (above, 2)):
        A, B, C = operands(dt, *shape)
        out, got = call(blx, dt, *shape, A, B, C)
        assert got == path
        native, _ = call(blx, dt, *shape, A, B, C, mode=1)
        # both within (K + 2) u (|alpha||A||B| + |beta||C|), complex products double
        u = 2.0 ** -53 * (2 if dt == "z" else 1)
        bound = 2 * (shape[2] + 2) * u * (1.5 * (B.abs() @ A.abs()) + 0.5 * C.abs())
        assert bool(((out - native).abs() <= bound).all())


@pytest.mark.parametrize("dt,shape", [("d", (1300, 1301, 1302)), ("z", (900, 901, 903))])
def test_wide_spread_and_no_scratch_take_the_native_kernel(blx, dt, shape):
    A, B, C = operands(dt, *shape, spread=6.0)
    out, path = call(blx, dt, *shape, A, B, C)
    native, _ = call(blx, dt, *shape, A, B, C, mode=1)
    assert path == 4 and torch.equal(out, native)
    A, B, C = operands(dt, *shape)
    native, _ = call(blx, dt, *shape, A, B, C, mode=1)
    blx.test_fail_allocation(1)
    out, path = call(blx, dt, *shape, A, B, C)
    blx.test_fail_allocation(0)
    assert path == 1 and torch.equal(out, native)
