"""Split TSMTTSM of operands that hold infinities or NaN: the entries of C that are not finite from the CUDA-core
kernels are NaN, all others agree; by the method's name, and where AUTO chooses it.  And of finite elements next to the largest number, whose column exponents have no headroom left."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [(4, 8, "auto"), (6, 6, "auto"), (4, 64, "auto"), (8, 8, "split"), (16, 16, "split"), (1, 1, "split"),
          (32, 32, "split"), (33, 20, "split"), (64, 64, "split"), (100, 70, "split")]


@pytest.mark.parametrize("M,N,acc", SHAPES)
@pytest.mark.parametrize("dt", [np.float64, np.float32, np.complex128, np.complex64])
@pytest.mark.parametrize("gram", [False, True])
def test_not_finite(handle, dt, M, N, acc, gram):
    cplx = np.dtype(dt).kind == "c"
    if cplx and max(M, N) > 64:
        pytest.skip("real width above 128")
    if acc == "auto" and dt in (np.float32, np.complex64):
        pytest.skip("AUTO is plain FP32")
    if acc == "auto" and gram and M * M < 32:
        pytest.skip("AUTO is plain FP64")
    N = M if gram else N
    K = (3 << 22) // (M * N) + 5 if acc == "auto" else 20003
    rng = np.random.default_rng(M + N)
    A0, B0 = common.uniform(rng, K * M, dt).reshape(K, M), common.uniform(rng, K * N, dt).reshape(K, N)
    for bad in (np.nan, np.inf, -np.inf, "two"):
        A, B = A0.copy(), B0.copy()
        (B if not gram and bad == np.inf else A)[K // 3, 0] = np.inf if bad == "two" else bad
        if bad == "two":  # opposite infinities in one column, far apart
            A[K - 2, 0] = -np.inf
        Ad = torch.from_numpy(A).cuda()
        Bd = Ad if gram else torch.from_numpy(B).cuda()
        out = []
        for a in (acc, "native"):
            C = torch.zeros(N, M, dtype=Ad.dtype, device="cuda")
            handle.tsmttsm(M, N, K, Ad, M, 1.0, Bd, N, 0.0, C, M, acc=a)
            out.append(torch.view_as_real(C).cpu().numpy() if cplx else C.cpu().numpy())
        got, exp = out
        assert not np.isfinite(exp).all()
        ok = np.isfinite(exp)
        assert np.array_equal(np.isnan(got), ~ok)
        assert np.abs(got[ok] - exp[ok]).max(initial=0.0) <= 2 * common.tol(dt, K) * K


@pytest.mark.parametrize("M,N", [(8, 8), (3, 5), (16, 16), (32, 32), (20, 40), (64, 64)])
def test_largest_exponents(handle, M, N):
    K = 5000
    rng = np.random.default_rng(M + N)
    r, c = np.arange(K)[:, None], np.arange(M)[None, :]
    A = rng.integers(-255, 256, (K, M)) * (1 << np.minimum((r // 16 + c) % 12, 5))  # |A| < 2^13
    B = rng.integers(-127, 128, (K, N))
    exp = (B.T @ A).astype(np.float64)
    Ad, Bd = torch.from_numpy(np.ldexp(A.astype(np.float64), 1010)).cuda(), torch.from_numpy(np.ldexp(B.astype(np.float64), -900)).cuda()
    C = torch.zeros(N, M, dtype=torch.float64, device="cuda")
    handle.tsmttsm(M, N, K, Ad, M, 1.0, Bd, N, 0.0, C, M, acc="split")
    assert np.array_equal(C.cpu().numpy(), np.ldexp(exp, 110))
