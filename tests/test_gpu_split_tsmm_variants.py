"""Split TSMM: each compiled variant (contraction width 16, 32, 64; 16 or 24 warps; with and without
old C) at the edges of its tiles: output widths that end inside a chunk of 4 columns and inside a
block, one to a few 128-row tiles per CTA and a short last one, more tiles than CTAs; beta zero (C
holds NaN), non-zero, folded in place; real and complex.  Bound: 8 sqrt(M) u normwise."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (M, N) real: width 16 with 16 warps, with 24 warps, width 32, width 64
REAL = [(16, 16), (5, 13), (16, 17), (9, 64), (12, 35), (17, 9), (32, 32), (33, 3), (64, 64), (50, 47)]
CPLX = [(8, 8), (3, 5), (8, 9), (7, 32), (16, 16), (9, 2), (32, 32), (20, 23)]


@pytest.mark.parametrize("dt,M,N", [(np.float64, *s) for s in REAL] + [(np.complex128, *s) for s in CPLX])
def test_variants(handle, dt, M, N):
    for K in (1, 127, 129, 2000, 152 * 128 * 2 + 77):
        rng = np.random.default_rng(M * 65 + N + K)
        A, B = common.uniform(rng, K * M, dt), common.uniform(rng, N * M, dt)
        for beta, inplace in ((0.0, False), (0.5, False), (0.5, True)):
            if inplace and M != N:
                continue
            C0 = A if inplace else common.uniform(rng, K * N, dt)
            C = torch.from_numpy(np.full(K * N, np.nan, dtype=dt) if beta == 0.0 else C0.copy()).cuda()
            handle.tsmm(M, N, K, C if inplace else torch.from_numpy(A).cuda(), M, 1.0, torch.from_numpy(B).cuda(), M, beta,
                        C, N, acc="split")
            exp, den = common.tsmm_expected(M, N, K, A, M, B, M, C0, N, 1.0, beta)
            assert common.normwise(C.cpu().numpy(), exp, den) <= common.tol(dt, M), (K, beta, inplace)
