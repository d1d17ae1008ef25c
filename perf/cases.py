"""Performance cases: the level-3 BLAS calls a user of blasx_b200 makes, through its public entry points.

Two ways of calling are covered: the device-resident entry points (`gemm_device`, `dsyrk_device`, `dtrsm_device`,
`dtrmm_device`; operands already on the GPU, as in a solver that keeps its matrices there) and the drop-in host calls
(`cblas_?gemm` on plain host arrays, copies included). All matrices are column-major: a matrix of `rows` x `cols` with
leading dimension `ld` is a torch tensor (or numpy array) of shape (cols, ld).

A case is a dict:
  kind    "gemm" (device-resident), "syrk", "trsm", "trmm" (device-resident, FP64), "host" (cblas_?gemm)
  dtype   "d" FP64, "s" FP32, "z" complex128, "c" complex64
  m, n, k sizes (syrk: C is n x n; trsm / trmm: B is m x n, k unused)
  ta, tb  "N", "T" or "C" (gemm); trans (the others); side, uplo, diag as in BLAS
  alpha, alpha_im, beta
  phi     entries are U[-0.5, 0.5] * exp(phi * g), g normal: 0 is well scaled, 4 spans many orders of magnitude
  pad     extra rows of every leading dimension
  pinned  host only: page-locked arrays instead of plain ones
"""
import math

import numpy as np
import torch

import blasx_b200 as bx

TORCH = {"d": torch.float64, "s": torch.float32, "z": torch.complex128, "c": torch.complex64}
ESIZE = {"d": 8, "s": 4, "z": 16, "c": 8}
CPLX = "zc"


def _gemm(name, dtype, ta, tb, m, n, k, alpha=1.0, beta=0.0, alpha_im=0.0, phi=0.0, pad=0, kind="gemm", pinned=False):
    c = {"kind": kind, "dtype": dtype, "ta": ta, "tb": tb, "m": m, "n": n, "k": k, "alpha": alpha,
         "alpha_im": alpha_im, "beta": beta, "phi": phi, "pad": pad}
    if kind == "host":
        c["pinned"] = pinned
    return {"name": name, **c} if name else c


def listed():
    return [
        # a tiny product inside an application's loop: the launch and the call are all there is
        _gemm("dgemm_small", "d", "N", "N", 96, 80, 64),
        # small single-precision and complex-single products, a few of them per step of a filter or a beamformer
        _gemm("sgemm_small", "s", "N", "T", 320, 257, 190),
        _gemm("cgemm_small", "c", "N", "C", 211, 300, 257, alpha=1.5, alpha_im=-0.5, beta=0.5),
        # the ordinary ragged FP64 call, below the size where the integer tensor cores pay
        _gemm("dgemm_ragged", "d", "T", "N", 1003, 777, 641, alpha=1.5, beta=-0.25),
        # an ordinary square FP64 call, e.g. a blocked factorisation's trailing update
        _gemm("dgemm_2048", "d", "N", "N", 2048, 2048, 2048, beta=0.5),
        # the benchmark of the library: the largest square FP64 product
        _gemm("dgemm_16384", "d", "N", "N", 16384, 16384, 16384, beta=0.5),
        # badly scaled data: the FP64 tensor pipe does the work
        _gemm("dgemm_wide", "d", "N", "N", 4096, 3000, 2500, beta=0.5, phi=4.0),
        # ragged FP32 and complex128 calls (the mixed-type benchmark's shapes at a tenth and a fifth)
        _gemm("sgemm_ragged", "s", "T", "N", 3001, 1777, 999, alpha=1.5, beta=-0.25),
        _gemm("zgemm_ragged", "z", "C", "C", 2401, 1639, 1203, alpha=1.5, alpha_im=0.5, beta=-0.25),
        # normal equations: a tall operand's Gram matrix
        {"name": "dsyrk_4000", "kind": "syrk", "dtype": "d", "uplo": "L", "trans": "N", "n": 4000, "k": 1000,
         "alpha": 1.0, "beta": 0.5, "phi": 0.0, "pad": 0},
        # a triangular system with many right-hand sides
        {"name": "dtrsm_4096", "kind": "trsm", "dtype": "d", "side": "L", "uplo": "U", "trans": "N", "diag": "N",
         "m": 4096, "n": 2048, "alpha": 1.0, "phi": 0.0, "pad": 0},
        # the drop-in call: plain host arrays, copied both ways
        _gemm("host_dgemm", "d", "N", "T", 1500, 1777, 1000, beta=0.5, kind="host"),
    ]


def _size(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.4:  # round sizes are as common as odd ones
        q = 64 if v >= 256 else 16
        v = max(q, v // q * q)
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["gemm"] * 6 + ["host", "syrk", "trsm", "trmm"])
    pad = rng.choice([0, 0, 0, 1, 8])
    if kind in ("gemm", "host"):
        dtype = rng.choice("dddssszc")
        top = 12000 if kind == "gemm" else 3000
        while True:
            m, n, k = (_size(rng, 48, top) for _ in range(3))
            if m * n * k * (4 if dtype in CPLX else 1) <= 1.5e11:
                break
        t = "NNTC" if dtype in CPLX else "NNT"
        alpha, beta = rng.choice([(1.0, 0.0), (1.0, 0.5), (1.5, -0.25), (-1.0, 1.0)])
        return _gemm(None, dtype, rng.choice(t), rng.choice(t), m, n, k, alpha=alpha, beta=beta,
                     alpha_im=rng.choice([0.0, 0.5]) if dtype in CPLX else 0.0,
                     phi=rng.choice([0.0, 0.0, 0.0, 1.0, 4.0]) if dtype in "dz" else rng.choice([0.0, 1.0]), pad=pad,
                     kind=kind, pinned=rng.random() < 0.5)
    if kind == "syrk":
        while True:
            n, k = _size(rng, 64, 8192), _size(rng, 64, 8192)
            if n * n * k <= 1.5e11:
                break
        return {"kind": "syrk", "dtype": "d", "uplo": rng.choice("UL"), "trans": rng.choice("NT"), "n": n, "k": k,
                "alpha": 1.0, "beta": rng.choice([0.0, 0.5]), "phi": 0.0, "pad": pad}
    while True:
        m, n = _size(rng, 64, 6000), _size(rng, 64, 6000)
        side = rng.choice("LR")
        if (m if side == "L" else n) ** 2 * (n if side == "L" else m) <= 1.5e11:
            break
    return {"kind": kind, "dtype": "d", "side": side, "uplo": rng.choice("UL"), "trans": rng.choice("NT"),
            "diag": rng.choice("NNU"), "m": m, "n": n, "alpha": rng.choice([1.0, -0.5]), "phi": 0.0, "pad": pad}


def _entries(shape, dtype, phi, gen):
    """U[-0.5, 0.5] * exp(phi g), drawn on the GPU."""
    real = torch.float64 if dtype in "dz" else torch.float32
    full = shape + ((2,) if dtype in CPLX else ())
    x = torch.rand(full, dtype=real, device="cuda", generator=gen) - 0.5
    if phi:
        x *= torch.exp(phi * torch.randn(full, dtype=real, device="cuda", generator=gen))
    return torch.view_as_complex(x) if dtype in CPLX else x


def _inputs(case, seed):
    """The operands as GPU tensors of shape (cols, ld), and their row counts."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt, pad, phi = case["dtype"], case["pad"], case["phi"]
    if case["kind"] in ("gemm", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        ra, ca = (m, k) if case["ta"] == "N" else (k, m)
        rb, cb = (k, n) if case["tb"] == "N" else (n, k)
        return {"A": (_entries((ca, ra + pad), dt, phi, gen), ra), "B": (_entries((cb, rb + pad), dt, phi, gen), rb),
                "C": (_entries((n, m + pad), dt, phi, gen), m)}
    if case["kind"] == "syrk":
        n, k = case["n"], case["k"]
        ra, ca = (n, k) if case["trans"] == "N" else (k, n)
        return {"A": (_entries((ca, ra + pad), dt, phi, gen), ra), "C": (_entries((n, n + pad), dt, phi, gen), n)}
    m, n = case["m"], case["n"]
    order = m if case["side"] == "L" else n
    A = _entries((order, order + pad), dt, phi, gen) / order
    A[:, :order].diagonal().add_(2.0)  # well conditioned
    return {"A": (A, order), "B0": (_entries((n, m + pad), dt, phi, gen), m)}


def prepare(case, seed):
    ops = _inputs(case, seed)
    s = {"case": case, **{name: t for name, (t, _) in ops.items()}, "rows": {name: r for name, (_, r) in ops.items()}}
    if case["kind"] == "host":
        for name in "ABC":
            h = s[name].cpu()
            s[name] = h.pin_memory() if case["pinned"] else h.numpy()
    if "B0" in s:
        s["B"] = torch.empty_like(s["B0"])
    return s


def _alpha(case):
    return complex(case["alpha"], case["alpha_im"]) if case["dtype"] in CPLX else case["alpha"]


def run(s):
    c = s["case"]
    kind, dt = c["kind"], c["dtype"]
    if kind == "gemm":
        A, B, C = s["A"], s["B"], s["C"]
        rc = bx.gemm_device(c["ta"], c["tb"], c["m"], c["n"], c["k"], _alpha(c), A, A.shape[1], B, B.shape[1],
                            c["beta"], C, C.shape[1], stream=torch.cuda.current_stream(), dtype=dt)
        out = C
    elif kind == "host":
        A, B, C = s["A"], s["B"], s["C"]
        call = {"d": bx.cblas_dgemm, "s": bx.cblas_sgemm, "z": bx.cblas_zgemm, "c": bx.cblas_cgemm}[dt]
        call(bx.CblasColMajor, bx.TRANS[c["ta"]], bx.TRANS[c["tb"]], c["m"], c["n"], c["k"], _alpha(c), A, A.shape[1],
             B, B.shape[1], c["beta"], C, C.shape[1])
        rc, out = bx.last_status(), C
    elif kind == "syrk":
        A, C = s["A"], s["C"]
        rc = bx.dsyrk_device(c["uplo"], c["trans"], c["n"], c["k"], c["alpha"], A, A.shape[1], c["beta"], C,
                             C.shape[1], stream=torch.cuda.current_stream())
        out = C
    else:  # in place: the right-hand sides (the factor) arrive in B, as the program before the call leaves them
        A, B = s["A"], s["B"]
        B.copy_(s["B0"])
        call = bx.dtrsm_device if kind == "trsm" else bx.dtrmm_device
        rc = call(c["side"], c["uplo"], c["trans"], c["diag"], c["m"], c["n"], c["alpha"], A, A.shape[1], B,
                  B.shape[1], stream=torch.cuda.current_stream())
        out = B
    if rc != 0:
        raise RuntimeError(bx.last_error())
    rows = s["rows"]["C" if "C" in s["rows"] else "B0"]
    return out[:, :rows]


def work(case):
    e = ESIZE[case["dtype"]]
    kind = case["kind"]
    if kind in ("gemm", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": e * (m * k + k * n + m * n * (2 if case["beta"] else 1)),
                "flops": (8.0 if case["dtype"] in CPLX else 2.0) * m * n * k}
    if kind == "syrk":
        n, k = case["n"], case["k"]
        return {"bytes": e * (n * k + n * (n + 1) / 2 * (2 if case["beta"] else 1)), "flops": float(n * (n + 1)) * k}
    m, n = case["m"], case["n"]
    order, vecs = (m, n) if case["side"] == "L" else (n, m)
    return {"bytes": e * (order * (order + 1) / 2 + 2 * m * n), "flops": float(order) * order * vecs}


def _op(x, t):
    """op of a column-major matrix held as its (cols, rows) tensor, as a rows x cols matrix."""
    return x.mT if t == "N" else (x.conj() if t == "C" else x)


def exact(case, seed):
    wide = torch.complex128 if case["dtype"] in CPLX else torch.float64
    ops = {name: t[:, :r].to(wide) for name, (t, r) in _inputs(case, seed).items()}
    kind = case["kind"]
    if kind in ("gemm", "host"):
        # alpha and beta as the call takes them: all values used here are exact in 32 bits
        out = _alpha(case) * (_op(ops["A"], case["ta"]) @ _op(ops["B"], case["tb"]))
        if case["beta"]:
            out += case["beta"] * ops["C"].mT
        out = out.mT
    elif kind == "syrk":
        X = _op(ops["A"], case["trans"])
        full = case["alpha"] * (X @ X.mT) + case["beta"] * ops["C"].mT
        keep = torch.ones_like(full, dtype=torch.bool)
        keep = keep.tril() if case["uplo"] == "L" else keep.triu()
        out = torch.where(keep, full, ops["C"].mT).mT
    else:
        A = ops["A"].mT
        A = A.tril() if case["uplo"] == "L" else A.triu()
        if case["diag"] == "U":
            A = A - torch.diag(A.diagonal()) + torch.eye(A.shape[0], dtype=wide, device=A.device)
        A = A if case["trans"] == "N" else A.mT
        B = case["alpha"] * ops["B0"].mT
        if kind == "trmm":
            out = (A @ B if case["side"] == "L" else B @ A).mT
        else:
            upper = (case["uplo"] == "U") == (case["trans"] == "N")
            out = torch.linalg.solve_triangular(A, B, upper=upper, left=case["side"] == "L").mT
    out = out.contiguous()
    return out.cpu().numpy() if kind == "host" and not case["pinned"] else out
