"""FP32 / complex FP32 TSMM on both sides of the rule that leaves shapes to the row-walking kernel: few outputs from
rows of up to 128 bytes (aligned or not), complex widths up to 6 x 2, and unaligned rows whose outputs do not fill the
cells; with and without beta, in place, columns out of a wide block.  Bounds as in test_gpu_tsmm_tile.py."""
import numpy as np
import pytest

from test_gpu_tsmm_tile import check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("M,N", [(8, 1), (8, 2), (8, 3), (9, 1), (9, 2), (9, 4), (12, 3), (6, 2), (4, 3), (7, 5), (16, 1),
                                 (17, 3), (15, 5), (16, 5), (17, 9), (31, 3), (33, 9)])
def test_either_side(handle, dt, M, N):
    for beta in (0.0, -0.5):
        for K in (3, 1025, 70001):
            check(handle, dt, M, N, K, M, N, beta=beta)
        check(handle, dt, M, N, 2049, M + 1, N + 1, beta=beta)
        check(handle, dt, M, N, 2049, 2 * M + 40, 2 * N + 40, beta=beta, shift=1)
        check(handle, dt, M, N, 2049, max(M, N) + 1, max(M, N) + 1, beta=beta, inplace=True)
