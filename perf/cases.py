"""The calls this library is measured on: tall-skinny products, SVQB and the request loop.

Each case is one pass through the public Python interface (`skinny_matmul_gb300.api`, a thin binding
of the C ABI), as a block solver or a service would make it.  The widths, row counts, types and
scalars are those of the benchmark's workloads (`bench.py`: C1's 8 x 8 Gram-like product, the TSMM
sweep at 1 GiB of A, the precision and SVQB workloads, the serving mix with K from 2^14 up, FP64 60 %,
complex FP64 25 %, FP32 15 %) and, between them, odd widths, odd row counts and padded leading
dimensions, which block solvers produce when vectors converge and are locked.

  listed()   the named cases            draw(rng)   one more of the same ranges
  prepare()  operands on the GPU        run()       one pass       exact()  its result in 64 bits
"""
import math
import random

import numpy as np
import torch

from skinny_matmul_gb300 import api

DTYPES = {"float32": torch.float32, "float64": torch.float64, "complex64": torch.complex64,
          "complex128": torch.complex128}
SIZE = {"float32": 4, "float64": 8, "complex64": 8, "complex128": 16}
SERVE_BUDGET = 8 << 30


def listed():
    return [
        # A solver's inner product of two small blocks on one rank's share of the rows: the smallest
        # call, all latency.  The method is the interface's default (plain FP64).
        {"name": "tsmttsm f64 4x4 short", "op": "tsmttsm", "dtype": "float64", "acc": "native", "M": 4, "N": 4,
         "K": 16384, "pad": 0, "gram": False, "conj": False, "alpha": 1.0, "beta": 0.0},
        # The benchmark's plain product: 8 x 8, 2^20 rows.
        {"name": "tsmttsm f64 8x8", "op": "tsmttsm", "dtype": "float64", "acc": "auto", "M": 8, "N": 8,
         "K": 1 << 20, "pad": 0, "gram": False, "conj": False, "alpha": 1.0, "beta": 0.0},
        # Projection of one block of 32 vectors on another (Rayleigh-Ritz), 2 GiB of operands.
        {"name": "tsmttsm f64 32x32", "op": "tsmttsm", "dtype": "float64", "acc": "auto", "M": 32, "N": 32,
         "K": 1 << 22, "pad": 0, "gram": False, "conj": False, "alpha": 1.0, "beta": 0.0},
        # A^H B of complex blocks after some vectors were locked: odd widths, odd row count.
        {"name": "tsmttsm c128 13x7 conj", "op": "tsmttsm", "dtype": "complex128", "acc": "auto", "M": 13, "N": 7,
         "K": 300007, "pad": 0, "gram": False, "conj": True, "alpha": 1.0, "beta": 0.0},
        # Single-precision blocks, accumulated into the result of an earlier call.
        {"name": "tsmttsm f32 16x16", "op": "tsmttsm", "dtype": "float32", "acc": "auto", "M": 16, "N": 16,
         "K": 1 << 21, "pad": 0, "gram": False, "conj": False, "alpha": 1.0, "beta": 0.5},
        # Gram matrix of a block in double-double accumulation: the check of an orthogonalisation.
        {"name": "gram f64 16 double-double", "op": "tsmttsm", "dtype": "float64", "acc": "dd", "M": 16, "N": 16,
         "K": 1 << 18, "pad": 0, "gram": True, "conj": False, "alpha": 1.0, "beta": 0.0},
        # The sweep's central shape: 16 x 16, 1 GiB of A, C accumulated with beta 0.5.
        {"name": "tsmm f64 16x16 1 GiB", "op": "tsmm", "dtype": "float64", "acc": "auto", "M": 16, "N": 16,
         "K": 1 << 23, "pad": 0, "inplace": False, "alpha": 1.0, "beta": 0.5},
        # Basis rotation in place: 64 vectors, 512 MiB.
        {"name": "tsmm f64 64 in place", "op": "tsmm", "dtype": "float64", "acc": "auto", "M": 64, "N": 64,
         "K": 1 << 20, "pad": 0, "inplace": True, "alpha": 1.0, "beta": 0.5},
        # Complex expansion of 8 vectors to 32 (the sweep's off-diagonal shape).
        {"name": "tsmm c128 8x32", "op": "tsmm", "dtype": "complex128", "acc": "auto", "M": 8, "N": 32,
         "K": 1 << 19, "pad": 0, "inplace": False, "alpha": 1.0, "beta": 0.5},
        # Single-precision restart: 20 vectors of a block that has room for more, cut to 12.
        {"name": "tsmm f32 20x12 padded", "op": "tsmm", "dtype": "float32", "acc": "auto", "M": 20, "N": 12,
         "K": 1000003, "pad": 12, "inplace": False, "alpha": 1.0, "beta": 0.0},
        # One step of a block iteration: the block times a small matrix, then SVQB of the result.
        {"name": "svqb f64 64", "op": "svqb", "dtype": "float64", "M": 64, "K": 1 << 19},
        # The request loop: a burst of 40 mixed products on operands resident in HBM.
        {"name": "serve 40 requests", "op": "serve", "requests": 40, "k_lo": 1 << 14, "k_hi": 1 << 18, "mix": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, hi):
    """Powers of two as often as any other width (odd ones among them), spread over their logarithm."""
    if rng.random() < 0.5:
        return 1 << rng.randint(0, int(math.log2(hi)))
    return _log_int(rng, 1, hi)


def draw(rng):
    kind = rng.choices(["tsmttsm", "tsmm", "svqb", "serve"], [45, 38, 10, 7])[0]
    if kind == "serve":
        return {"op": "serve", "requests": rng.randint(8, 60), "k_lo": 1 << 14, "k_hi": 1 << rng.randint(15, 18),
                "mix": rng.randint(2, 1 << 20)}
    if kind == "svqb":
        M = rng.choice([4, 8, 16, 24, 32, 48, 64, rng.randint(3, 63)])
        return {"op": "svqb", "dtype": "float64", "M": M, "K": _log_int(rng, 1 << 14, (1 << 25) // M)}
    dtype = rng.choices(["float64", "complex128", "float32", "complex64"], [57, 24, 14, 5])[0]
    cplx = dtype.startswith("complex")
    hi = 64 if kind == "tsmm" or dtype != "float64" else 128
    M, N = _width(rng, hi), _width(rng, hi)
    acc = rng.choices(["auto", "native", "dd"], [75, 18, 7])[0]
    if acc == "dd" and dtype != "float64":
        acc = "auto"
    same = rng.random() < 0.2  # a Gram matrix, or in place
    if same or rng.random() < 0.4:
        N = M
    pad = rng.choice([0, 0, 0, 1, 4, 12])
    s = SIZE[dtype]
    # at most about 1 GB of operands; plain and double-double products are bound by arithmetic
    most = (1 << 30) // (s * (M + pad + 2 * N))
    fma = M * N * (4 if cplx else 1)
    if acc == "dd":
        most = min(most, (1 << 27) // fma)
    elif acc == "native" and dtype in ("float64", "complex128"):
        most = min(most, (1 << 31) // fma)
    K = _log_int(rng, 1 << 13, max(1 << 13, min(1 << 24, most)))
    if rng.random() < 0.4:
        K -= K % 1024  # round row counts beside odd ones
    case = {"op": kind, "dtype": dtype, "acc": acc, "M": M, "N": N, "K": K, "pad": pad,
            "alpha": rng.choice([1.0, 1.0, -1.0, 0.75]), "beta": rng.choice([0.0, 0.0, 0.5])}
    if kind == "tsmttsm":
        case.update(gram=same, conj=cplx and rng.random() < 0.5)
    else:
        case.update(inplace=same)
        if same:
            case.update(alpha=1.0, beta=0.5)
    return case


# ------------------------------------------------------------------------------------- operands
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, rows, cols, dtype):
    """rows x cols of U[-1, 1)."""
    if dtype.is_complex:
        real = torch.float32 if dtype == torch.complex64 else torch.float64
        return torch.view_as_complex(torch.rand(rows, cols, 2, generator=g, device="cuda", dtype=real).mul_(2).sub_(1))
    return torch.rand(rows, cols, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _orthogonal(seed, M, dtype):
    """A seeded orthogonal (unitary) M x M matrix in 64 bits."""
    r = np.random.default_rng(seed)
    z = r.standard_normal((M, M))
    if dtype.is_complex:
        z = z + 1j * r.standard_normal((M, M))
    return torch.from_numpy(np.linalg.qr(z)[0])


def _requests(case):
    """The burst's products: TSMTTSM and TSMM, widths, types and K drawn as the serving workload draws them."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["requests"]):
        op = rng.choices(["tsmttsm", "tsmm"], [50, 35])[0]
        dtype = rng.choices(["float64", "complex128", "float32"], [60, 25, 15])[0]
        M, N = (rng.choice([1, 2, 4, 8, 16, 32, 64]) for _ in range(2))
        out.append((op, dtype, M, N, _log_int(rng, case["k_lo"], case["k_hi"])))
    return out


_server = None


def _the_server():
    """The request loop of this process: one server, kept as a service keeps it."""
    global _server
    if _server is None:
        _server = api.Server(api.default_handle(), SERVE_BUDGET, num_streams=8, max_inflight=16)
    return _server


def prepare(case, seed):
    g = _gen(seed)
    h = api.default_handle()
    if case["op"] == "serve":
        reqs = []
        for op, dtype, M, N, K in _requests(case):
            dt = DTYPES[dtype]
            A = _uniform(g, K, M, dt)
            if op == "tsmttsm":
                B, C = _uniform(g, K, N, dt), torch.zeros(N, M, dtype=dt, device="cuda")
            else:
                B, C = _uniform(g, N, M, dt), torch.zeros(K, N, dtype=dt, device="cuda")
            reqs.append((op, dtype, M, N, K, A, B, C))
        return {"case": case, "server": _the_server(), "reqs": reqs}
    dt = DTYPES[case["dtype"]]
    M, K = case["M"], case["K"]
    if case["op"] == "svqb":
        V = torch.randn(K, M, generator=g, device="cuda", dtype=dt)
        # the small matrix: singular values log-spaced from 1 to 1/10 between two orthogonal factors
        sig = torch.logspace(0, -1, M, dtype=torch.float64)
        W = _orthogonal(seed, M, dt) @ torch.diag(sig) @ _orthogonal(seed + 1, M, dt).T
        return {"case": case, "h": h, "V": V, "W": W.T.contiguous().cuda(), "X": torch.empty_like(V)}
    N, pad = case["N"], case["pad"]
    A = _uniform(g, K, M + pad, dt)
    if case["op"] == "tsmttsm":
        B = A if case["gram"] else _uniform(g, K, N, dt)
        C = _uniform(g, N, M, dt)
    elif case["inplace"]:
        # alpha A B + beta A = A Q with an orthogonal Q: the basis keeps its length over many steps
        Q = _orthogonal(seed, M, dt) - case["beta"] * torch.eye(M, dtype=torch.float64)
        B, C = Q.to(dt).cuda(), A
    else:
        B, C = _uniform(g, N, M, dt), _uniform(g, K, N, dt)
    return {"case": case, "h": h, "A": A, "B": B, "C": C}


def run(state):
    c = state["case"]
    if c["op"] == "serve":
        s = state["server"]
        tickets = [s.submit(op, dtype, M, N, K, A, M, B, N if op == "tsmttsm" else M, C, M if op == "tsmttsm" else N,
                            acc="auto", device=True)[1] for op, dtype, M, N, K, A, B, C in state["reqs"]]
        for t in tickets:
            if s.wait(t) != (0, 0):
                raise RuntimeError("a request failed")
        return [q[7] for q in state["reqs"]]
    h, M, K = state["h"], c["M"], c["K"]
    if c["op"] == "svqb":
        h.tsmm(M, M, K, state["V"], M, 1.0, state["W"], M, 0.0, state["X"], M, acc="auto")
        h.svqb(K, M, state["X"], M, orth_err=False)
        return state["X"]
    A, B, C, N, lda = state["A"], state["B"], state["C"], c["N"], M + c["pad"]
    if c["op"] == "tsmttsm":
        h.tsmttsm(M, N, K, A, lda, c["alpha"], B, lda if c["gram"] else N, c["beta"], C, M, acc=c["acc"], conj=c["conj"])
    else:
        h.tsmm(M, N, K, A, lda, c["alpha"], B, M, c["beta"], C, lda if c["inplace"] else N, acc=c["acc"])
    return C


def _product_work(op, dtype, M, N, K, reads_b=True, reads_c=False):
    s = SIZE[dtype]
    f = 8 if dtype.startswith("complex") else 2
    if op == "tsmttsm":
        return s * (K * (M + (N if reads_b else 0)) + M * N * (2 if reads_c else 1)), f * M * N * K
    return s * (K * (M + N * (2 if reads_c else 1)) + M * N), f * M * N * K


def work(case):
    """Bytes: each input read once, each output written once.  Flops: those of the plain product."""
    if case["op"] == "serve":
        parts = [_product_work(*q) for q in _requests(case)]
    elif case["op"] == "svqb":
        # V once and the result once: the small transforms could in principle be applied together
        M, K = case["M"], case["K"]
        parts = [_product_work("tsmm", "float64", M, M, K), (0, 4 * M * M * K)]
    else:
        parts = [_product_work(case["op"], case["dtype"], case["M"], case["N"], case["K"], reads_b=not case.get("gram"),
                               reads_c=case["beta"] != 0.0 and not case.get("inplace"))]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# --------------------------------------------------------------------------------------- exact
def _wide(x):
    return x.to(torch.complex128 if x.dtype.is_complex else torch.float64)


def _exact_tsmttsm(A, B, conj=False):
    """sum_k A[k, m] B[k, n] stored [n, m], in chunks of rows so that partial sums stay short."""
    out = 0
    for k in range(0, A.shape[0], 1 << 16):
        a, b = _wide(A[k:k + (1 << 16)]), _wide(B[k:k + (1 << 16)])
        out = out + b.T @ (a.conj() if conj else a)
    return out


def exact(case, seed):
    st = prepare(case, seed)
    if case["op"] == "serve":
        return [_exact_tsmttsm(A, B) if op == "tsmttsm" else _wide(A) @ _wide(B).T
                for op, dtype, M, N, K, A, B, C in st["reqs"]]
    M = case["M"]
    if case["op"] == "svqb":
        X = st["V"] @ st["W"].T
        S = _exact_tsmttsm(X, X).T
        d = torch.diagonal(S).rsqrt()
        lam, U = torch.linalg.eigh((S * d[:, None] * d[None, :]).cpu())
        U = U * torch.sign(U[U.abs().argmax(dim=0), torch.arange(M)])[None, :]
        T = d.cpu()[:, None] * U / lam.clamp_min(1e-15).sqrt()[None, :]
        return X @ T.cuda()
    A, B, C = st["A"], st["B"], st["C"]
    if case["op"] == "tsmttsm":
        P = _exact_tsmttsm(A[:, :M], B[:, :case["N"]], case["conj"])
        return case["alpha"] * P + case["beta"] * _wide(C)
    P = case["alpha"] * (_wide(A[:, :M]) @ _wide(B).T)
    if case["inplace"]:  # only the first M columns of a padded block change
        return torch.cat([P + case["beta"] * _wide(A[:, :M]), _wide(A[:, M:])], dim=1)
    return P + case["beta"] * _wide(C)
