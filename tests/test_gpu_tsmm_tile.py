"""The tiled FP32 / complex FP32 TSMM at the edges of its tiles.

Widths around 16 bytes of a row (4 floats, 2 complex numbers), one column on either side, widths
that leave part of the last vector, the widest in and out and one whose ring does not fit (left to the row kernel);
row counts of one tile pass and around it, a few rows, and enough for several tiles per CTA; dense,
padded by a vector, padded by one element (element copies and stores), unaligned starts, in place
(folded, padded and with M != N), beta with values that must not be read (NaN, beta = 0).
Bounds: 8 sqrt(M) u normwise (u = 2^-24), and the columns beside the outputs untouched."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WIDTHS = [(5, 1), (1, 5), (4, 5), (8, 8), (7, 9), (13, 13), (20, 12), (33, 31), (64, 64), (64, 1), (3, 64), (128, 96)]


def check(handle, dt, M, N, K, lda, ldc, alpha=1.5, beta=-0.5, inplace=False, shift=0):
    rng = np.random.default_rng(M * 131 + N * 7 + K)
    A = common.uniform(rng, K * lda, dt)
    B = common.uniform(rng, N * M, dt)
    C0 = A if inplace else common.uniform(rng, K * ldc, dt)
    if beta == 0 and not inplace:
        C0 = np.full(K * ldc, np.nan, dtype=dt)

    def dev(x):  # `shift` elements past an aligned start
        t = torch.empty(x.size + shift, dtype=torch.from_numpy(x).dtype, device="cuda")[shift:]
        return t.copy_(torch.from_numpy(x))
    Ad, Bd = dev(A), dev(B)
    Cd = Ad if inplace else dev(C0)
    handle.tsmm(M, N, K, Ad, lda, alpha, Bd, M, beta, Cd, ldc, acc="native")
    got = Cd.cpu().numpy()
    wide = np.complex128 if np.dtype(dt).kind == "c" else np.float64
    exp, den = common.tsmm_expected(M, N, K, A.astype(wide), lda, B.astype(wide), M, np.nan_to_num(C0).astype(wide), ldc,
                                    alpha, beta)
    mask = common.c_mask_tsmm(N, K, ldc)
    assert common.normwise(got, exp, den, mask) <= common.tol(dt, max(M, 1))
    assert np.array_equal(got[~mask], C0[~mask], equal_nan=True)


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("M,N", WIDTHS)
def test_tile_edges(handle, dt, M, N):
    for K in (1, 31, 257, 3001):
        check(handle, dt, M, N, K, M, N)
    check(handle, dt, M, N, 2049, M + 4, N + 4, beta=0.0)
    check(handle, dt, M, N, 2049, M + 1, N + 3)
    check(handle, dt, M, N, 1025, M, N, shift=1)


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("M,N,ld", [(8, 8, 8), (13, 13, 16), (20, 12, 24), (12, 20, 24), (64, 64, 64)])
def test_in_place(handle, dt, M, N, ld):
    for K in (1, 300, 70001):
        check(handle, dt, M, N, K, ld, ld, alpha=0.75, beta=0.5, inplace=True)
        check(handle, dt, M, N, K, ld, ld, alpha=1.0, beta=0.0, inplace=True)
