"""GPU tests of the native kernels, one shape per tile and per k cut, with the
launched kernel and its grid read back: the choice itself is tested, and the
products of small integers are exact. k spans several turns of each tile's ring
of stages."""
import json
import os
import re
import tempfile

import pytest
import torch

pytestmark = pytest.mark.gpu

T = {"d": torch.float64, "s": torch.float32, "z": torch.complex128, "c": torch.complex64}


def launched(fn):
    """(kernel name, blocks) of the native GEMM kernels that fn launches."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        p.export_chrome_trace(os.path.join(d, "trace.json"))
        with open(os.path.join(d, "trace.json")) as f:
            events = json.load(f)["traceEvents"]
    return [(e["name"], e["args"]["grid"][0]) for e in events
            if e.get("cat") == "kernel" and re.search(r"dmma_|fma_|sgemm128", e["name"])]


def tile_of(name):
    """The C tile of a native kernel, from its template arguments."""
    m = re.search(r"dmma_\w+_kernel<(true|false), (?:true|false), (?:true|false), \d+, (\d)>", name)
    if m:
        g = int(m[2])
        return {0: (64, 128) if m[1] == "true" else (128, 128), 1: (64, 64), 2: (32, 32), 3: (64, 48)}[g]
    if "sgemm128" in name:
        return 128, 128
    m = re.search(r"FmaTile<[^,]+, (\d+), (\d+), (\d+), ", name)
    return 32 * int(m[1]), 32 * int(m[2])


def integers(gen, rows, ld, dt, top):
    x = torch.randint(-top, top + 1, (rows, ld), device="cuda", generator=gen, dtype=torch.int32)
    if dt in "zc":
        return torch.complex(x.to(torch.float64), torch.randint(-top, top + 1, (rows, ld), device="cuda", generator=gen,
                                                                dtype=torch.int32).to(torch.float64)).to(T[dt])
    return x.to(T[dt])


@pytest.fixture
def native(blx):
    prev = blx.set_dgemm_mode(blx.MODE_NATIVE)
    yield blx
    blx.set_dgemm_mode(prev)


def op(x, t):
    return x.mT if t == "N" else (x.conj() if t == "C" else x)


def run(blx, dt, ta, tb, m, n, k, pad, tile, cut, beta=-1.0):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n + k)
    top = 2 if dt in "sc" else 8  # sums below 2^24 (2^53)
    ra, ca = (m, k) if ta == "N" else (k, m)
    rb, cb = (k, n) if tb == "N" else (n, k)
    A, B, C = integers(gen, ca, ra + pad, dt, top), integers(gen, cb, rb + pad, dt, top), integers(gen, n, m + pad, dt, top)
    out = C.clone()

    def call():
        rc = blx.gemm_device(ta, tb, m, n, k, 2.0, A, ra + pad, B, rb + pad, beta, out, m + pad, dtype=dt)
        assert rc == blx.BLASX_OK, blx.last_error()

    kernels = launched(call)
    assert len(kernels) == 1, kernels
    name, blocks = kernels[0]
    assert tile_of(name) == tile, name
    tiles = -(-m // tile[0]) * (1 if "sgemm128" in name else -(-n // tile[1]))  # (the grid's first extent)
    assert blocks == tiles * cut and ("split" in name) == (cut > 1), (name, blocks, tiles)
    wide = torch.complex128 if dt in "zc" else torch.float64
    want = C.to(wide).clone()
    want[:, :m] = (2 * (op(A[:, :ra].to(wide), ta) @ op(B[:, :rb].to(wide), tb)) + beta * C[:, :m].to(wide).mT).mT
    assert torch.equal(out.to(wide), want)


@pytest.mark.parametrize("ta,tb,tile", [("N", "N", (64, 64)), ("C", "C", (64, 64)), ("N", "T", (64, 64)),
                                        ("T", "N", (32, 32)), ("C", "N", (32, 32))])
@pytest.mark.parametrize("shape", [(1408, 1664, 500), (1471, 1599, 83)])
def test_complex128_tiles_by_layout(native, ta, tb, tile, shape):
    run(native, "z", ta, tb, *shape, 0, tile, 1)


@pytest.mark.parametrize("ta,tb,shape,pad,tile", [
    ("N", "T", (1000, 1000, 1000), 0, (32, 32)), ("N", "T", (1000, 1000, 1000), 1, (64, 64)),  # 8-byte copies
    ("T", "T", (1000, 1000, 1000), 1, (64, 64)), ("N", "N", (1000, 1000, 1000), 1, (64, 64)),
    ("N", "T", (1003, 777, 641), 0, (32, 32)),
    ("N", "N", (1003, 777, 641), 0, (64, 48)),
])
def test_fp64_tiles_by_copy_width(native, ta, tb, shape, pad, tile):
    run(native, "d", ta, tb, *shape, pad, tile, 1)


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("shape,pad,tile", [((2500, 2492, 300), 1, (128, 128)), ((2500, 2492, 300), 0, (64, 64)),
                                            ((2170, 2165, 257), 0, (128, 128)), ((2100, 2150, 192), 1, (128, 128)),
                                            ((2100, 2150, 191), 1, (64, 64)),
                                            ((2400, 2400, 300), 1, (64, 64))])
def test_fp32_tiles_by_copy_width(native, ta, tb, shape, pad, tile):
    m, n, k = shape
    run(native, "s", ta, tb, m, n, k, pad, tile, 1)


@pytest.mark.parametrize("ta,tb,shape,pad,tile", [
    ("N", "N", (2100, 2150, 96), 1, (128, 128)), ("T", "N", (2100, 2150, 95), 1, (64, 64)),
    ("N", "T", (2100, 2150, 96), 0, (128, 128)), ("N", "T", (2100, 2150, 95), 0, (64, 64)),  # op(B) alone narrow
    ("N", "N", (2100, 2152, 300), 0, (64, 64)),
])
def test_fp32_tiles_without_c(native, ta, tb, shape, pad, tile):
    run(native, "s", ta, tb, *shape, pad, tile, 1, beta=0.0)


def test_fp32_large_tile_as_the_fallback(blx):
    # operands of wide spread with odd leading dimensions: the decision on the
    # device leaves the call to the native kernel, bit for bit
    m, n, k = 2170, 2165, 300
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)

    def wide(cols, ld):
        x = torch.rand((cols, ld), device="cuda", generator=gen) - 0.5
        return x * torch.exp(6 * torch.randn((cols, ld), device="cuda", generator=gen))

    A, B, C = wide(k, m + 1), wide(n, k + 1), wide(n, m + 1)
    outs = []
    for mode, path in ((blx.MODE_AUTO, 4), (blx.MODE_NATIVE, 1)):
        prev = blx.set_dgemm_mode(mode)
        out = C.clone()
        kernels = launched(lambda: blx.gemm_device("N", "N", m, n, k, 1.5, A, m + 1, B, k + 1, -0.5, out, m + 1, dtype="s"))
        blx.set_dgemm_mode(prev)
        assert blx.call_stats()["path"] == path
        assert tile_of(kernels[-1][0]) == (128, 128)
        outs.append(out)
    assert torch.equal(*outs)


@pytest.mark.parametrize("dt,ta,tb,shape,pad,tile,cut", [
    ("d", "N", "N", (1408, 1664, 500), 0, (128, 128), 1), ("d", "T", "N", (1408, 1664, 500), 0, (128, 128), 1),
    ("d", "N", "T", (1408, 1664, 500), 1, (128, 128), 1),
    ("d", "N", "N", (1300, 1301, 1302), 0, (64, 64), 1), ("d", "T", "T", (1300, 1301, 1302), 1, (64, 64), 1),
    ("d", "T", "T", (951, 2478, 338), 1, (64, 64), 1),  # two CTAs per SM
    ("d", "T", "N", (1003, 777, 641), 0, (64, 48), 1), ("d", "N", "T", (300, 257, 60), 0, (32, 32), 1),
    ("d", "T", "N", (35, 59, 253), 0, (32, 32), 4), ("d", "N", "N", (300, 299, 500), 1, (32, 32), 4),
    ("d", "N", "T", (30, 32, 261), 0, (32, 32), 8), ("d", "T", "T", (100, 130, 300), 1, (32, 32), 8),
    ("d", "N", "N", (96, 64, 1990), 0, (32, 32), 16), ("d", "T", "N", (33, 31, 700), 1, (32, 32), 16),
    ("z", "T", "T", (41, 30, 133), 0, (32, 32), 4), ("z", "N", "N", (100, 130, 300), 0, (32, 32), 8),
    ("z", "C", "N", (100, 130, 300), 1, (32, 32), 8), ("z", "N", "T", (160, 160, 700), 0, (32, 32), 16),
    ("z", "C", "C", (200, 190, 700), 1, (32, 32), 16), ("z", "N", "N", (300, 300, 100), 0, (32, 32), 1),
    ("s", "N", "N", (320, 257, 190), 0, (32, 32), 1), ("s", "T", "T", (700, 640, 128), 1, (32, 32), 1),
    ("s", "T", "N", (1400, 1300, 333), 0, (64, 64), 1), ("s", "N", "T", (1400, 1300, 333), 1, (64, 64), 1),
    ("s", "N", "N", (64, 96, 600), 0, (32, 32), 2), ("s", "T", "N", (61, 95, 1100), 1, (32, 32), 4),
    ("s", "N", "T", (64, 96, 2100), 0, (32, 32), 8), ("s", "T", "T", (61, 95, 4200), 0, (32, 32), 16),
    ("c", "N", "N", (500, 500, 60), 0, (32, 32), 1), ("c", "C", "T", (600, 620, 100), 1, (32, 32), 1),
    ("c", "N", "C", (64, 96, 130), 0, (32, 32), 2), ("c", "T", "N", (211, 300, 257), 1, (32, 32), 4),
    ("c", "C", "N", (61, 95, 520), 0, (32, 32), 8), ("c", "N", "T", (64, 96, 1030), 0, (32, 32), 16),
])
def test_every_tile_and_cut(native, dt, ta, tb, shape, pad, tile, cut):
    run(native, dt, ta, tb, *shape, pad, tile, cut)


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n,k,trans,tile", [(1901, 300, "N", (128, 128)), (1355, 300, "N", (64, 64)), (1537, 300, "N", (64, 48)),
                                            (1089, 300, "T", (64, 48)), (1348, 91, "T", (64, 64)), (2118, 90, "T", (128, 128)),
                                            (300, 300, "N", (32, 32)), (200, 700, "T", (32, 32))])
def test_triangular_output(native, uplo, n, k, trans, tile):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    rows, cols = (n, k) if trans == "N" else (k, n)
    A, C = integers(gen, cols, rows, "d", 8), integers(gen, n, n, "d", 8)
    out = C.clone()

    def call():
        rc = native.dsyrk_device(uplo, trans, n, k, 2.0, A, rows, -1.0, out, n)
        assert rc == native.BLASX_OK, native.last_error()

    kernels = launched(call)
    assert len(kernels) == 1 and tile_of(kernels[0][0]) == tile, kernels
    X = op(A, trans)
    full = 2 * (X @ X.mT) - C.mT
    keep = torch.ones_like(full, dtype=torch.bool)
    keep = keep.tril() if uplo == "L" else keep.triu()
    assert torch.equal(out, torch.where(keep, full, C.mT).mT)
