"""The CUDA-core TSMTTSM at the edges of its register tiles, row slices and reductions.

Widths that leave edge cells on every side of a 1 x 1 .. 8 x 8 tile, one cell only, a full group of
256 cells and more than one group; row counts around one row tile (16 rows), one tile per CTA, and
enough rows for a second CTA per SM and for the two-level sum of the CTA partials; dense, padded
(element copies) and Gram operands, whose mirrored half is checked against the oracle like the rest.
Bounds: 8 sqrt(K) u normwise (double-double: the output rounding, 2^-52 FP64 and 2^-51 complex)."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WIDTHS = [(1, 1), (1, 64), (3, 2), (7, 7), (9, 8), (13, 7), (17, 16), (20, 12), (33, 5), (48, 40), (64, 64), (65, 68)]
KINDS = [(np.float32, "native"), (np.float64, "native"), (np.complex64, "native"), (np.complex128, "native"),
         (np.float64, "dd"), (np.complex128, "dd")]


def check(handle, dt, acc, M, N, K, gram=False, conj=False, pad=0, beta=0.5):
    rng = np.random.default_rng(M * 100 + N + K)
    lda, ldb, ldc = M + pad, (M if gram else N) + pad, M + 1
    A = common.uniform(rng, K * lda, dt)
    B = A if gram else common.uniform(rng, K * ldb, dt)
    C0 = common.uniform(rng, N * ldc, dt)
    Ad = torch.from_numpy(A).cuda()
    Bd = Ad if gram else torch.from_numpy(B).cuda()
    Cd = torch.from_numpy(C0.copy()).cuda()
    handle.tsmttsm(M, N, K, Ad, lda, 1.5, Bd, ldb, beta, Cd, ldc, acc=acc, conj=conj)
    got = Cd.cpu().numpy()
    wide = np.complex128 if np.dtype(dt).kind == "c" else np.float64
    exp, den = common.tsmttsm_expected(M, N, K, (A.conj() if conj else A).astype(wide), lda, B.astype(wide), ldb,
                                       C0.astype(wide), ldc, 1.5, beta)
    mask = common.c_mask_tsmttsm(M, N, ldc)
    bound = {np.float64: 2.0 ** -52, np.complex128: 2.0 ** -51}[dt] if acc == "dd" else common.tol(dt, K)
    assert common.normwise(got, exp, den, mask) <= bound
    assert np.array_equal(got[~mask], C0[~mask]), "only C's own entries are written"


@pytest.mark.parametrize("M,N", WIDTHS)
@pytest.mark.parametrize("dt,acc", KINDS, ids=lambda x: str(x))
def test_tile_edges(handle, dt, acc, M, N):
    for K in (1, 16, 17, 1000, 5003) if acc == "native" else (17, 1000):
        check(handle, dt, acc, M, N, K)
        check(handle, dt, acc, M, N, K, pad=3, beta=0.0)


@pytest.mark.parametrize("M", [1, 4, 7, 8, 12, 17, 32, 64])
@pytest.mark.parametrize("dt,acc", KINDS, ids=lambda x: str(x))
def test_gram_mirror(handle, dt, acc, M):
    for K in (15, 4099):
        check(handle, dt, acc, M, M, K if acc == "native" else min(K, 500), gram=True)
    if np.dtype(dt).kind == "c" and acc == "native":
        check(handle, dt, acc, M, M, 4099, gram=True, conj=True)


@pytest.mark.parametrize("M,N,K", [(16, 16, 45003), (13, 7, 80001), (8, 8, 250007), (20, 12, 40005)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_many_ctas_and_two_levels(handle, dt, M, N, K):
    check(handle, dt, "native", M, N, K)
    check(handle, dt, "native", M, M, K, gram=True)
