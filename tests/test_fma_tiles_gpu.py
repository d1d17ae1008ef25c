"""GPU tests of the native FP32 / complex64 tiles: tile edges and remainders,
every copy width, the k extent cut over groups of warps and over a cluster.

Small integers whose products and sums stay below 2^24 make every order of
summation exact, so the comparison is for equality.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# one 32x32 tile and its edges with k cuts up to 16; both 32x32 forms; the 64x64 FP32 form; remainders in every direction
SHAPES = [(1, 1, 1), (31, 33, 65), (32, 32, 512), (33, 31, 4100), (96, 64, 1030), (65, 47, 33), (400, 300, 150),
          (700, 600, 37), (1500, 1301, 20)]


@pytest.fixture
def native(blx):
    prev = blx.set_dgemm_mode(blx.MODE_NATIVE)
    yield blx
    blx.set_dgemm_mode(prev)


def on_gpu(x, offset):
    """x's bytes on the GPU, starting `offset` floats past a 16-byte boundary."""
    flat = torch.from_numpy(x.reshape(-1).view(np.float32))
    buf = torch.zeros(flat.numel() + 4, dtype=torch.float32, device="cuda")
    buf[offset:offset + flat.numel()] = flat.cuda()
    return buf, buf.data_ptr() + 4 * offset


@pytest.mark.parametrize("dt", ["s", "c"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("C", "C")])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("pad,offset", [(0, 0), (1, 0), (0, 1), (2, 2)])
def test_tiles_are_exact_on_integers(native, blx, dt, ta, tb, shape, pad, offset):
    M, N, K = shape
    rng = np.random.default_rng(M * 31 + N * 7 + K)

    def stored(rows, cols):
        x = rng.integers(-20, 21, (cols, rows + pad)).astype(np.float32)
        return x if dt == "s" else (x + 1j * rng.integers(-20, 21, x.shape)).astype(np.complex64)

    A = stored(*((M, K) if ta == "N" else (K, M)))
    B = stored(*((K, N) if tb == "N" else (N, K)))
    C = stored(M, N)

    def op(x, t):
        x = x[:, :x.shape[1] - pad].astype(np.complex128 if dt == "c" else np.float64)
        return x.T if t == "N" else (x.conj() if t == "C" else x)

    want = C.copy()
    want[:, :M] = (2 * (op(A, ta) @ op(B, tb)) - 3 * C[:, :M].T).T
    keep_a, pa = on_gpu(A, offset)
    keep_b, pb = on_gpu(B, offset)
    dC, pc = on_gpu(C, offset)
    rc = blx.gemm_device(ta, tb, M, N, K, 2.0, pa, A.shape[1], pb, B.shape[1], -3.0, pc, M + pad, dtype=dt)
    assert rc == blx.BLASX_OK, blx.last_error()
    got = dC.cpu().numpy()[offset:offset + C.size * (2 if dt == "c" else 1)].view(C.dtype).reshape(C.shape)
    np.testing.assert_array_equal(got, want)
