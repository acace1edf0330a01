"""CUDA-core TSMTTSM of FP32 and complex FP32 storage, plain and summed in FP64: operands that are columns of a wide
block (no bulk copies) or whole ones, on both sides of the row counts where the row-streaming kernel and the ring
kernel take over from one another.  Against numpy in FP64; bounds: 8 sqrt(K) 2^-24 normwise for FP32 sums,
2^-23 (one rounding) for FP64 sums."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("acc,K", [("native", 3001), ("native", (1 << 20) - 1), ("native", 1 << 20),
                                   ("native", 3 << 19), ("dd", 4096), ("dd", (1 << 16) - 1), ("dd", 1 << 16),
                                   ("dd", (1 << 17) - 1), ("dd", 1 << 17)])
@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("M,N,gram", [(5, 3, False), (8, 4, False), (6, 7, False), (8, 8, False), (6, 6, True),
                                      (7, 7, True), (8, 8, True)])
def test_columns_of_a_block(handle, dt, acc, K, M, N, gram):
    rng = np.random.default_rng(M * 10 + N)
    for wide in (0, 44) if K < 1 << 18 else (44,) if M == 6 else (0,):
        ld, c0 = max(M, N) + wide, 1 if wide else 0
        X = common.uniform(rng, K * ld, dt).reshape(K, ld)
        Y = X if gram else common.uniform(rng, K * ld, dt).reshape(K, ld)
        Xd = torch.from_numpy(X).cuda()
        Yd = Xd if gram else torch.from_numpy(Y).cuda()
        C = torch.zeros(N, M, dtype=Xd.dtype, device="cuda")
        s, code = Xd.element_size(), 0 if dt == np.float32 else 2
        handle.tsmttsm(M, N, K, Xd.data_ptr() + c0 * s, ld, 1.0, Yd.data_ptr() + c0 * s, ld, 0.0, C, M, acc=acc, dtype=code)
        up = np.complex128 if dt == np.complex64 else np.float64
        a, b = X[:, c0:c0 + M].astype(up), Y[:, c0:c0 + N].astype(up)
        err = np.linalg.norm(C.cpu().numpy() - b.T @ a) / np.linalg.norm(np.abs(b).T @ np.abs(a))
        assert err <= (common.tol(dt, K) if acc == "native" else 2.0**-23)
