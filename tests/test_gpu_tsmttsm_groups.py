"""The CUDA-core TSMTTSM with more than 256 cells: several groups of cells (gridDim.y), the last of which
has fewer cells, hence several row slices and the largest reduction in shared memory.  Bounds as in
test_gpu_tsmttsm_tiles.py; FP32 in double-double accumulates in FP64 and is rounded once."""
import numpy as np
import pytest

import common
from test_gpu_tsmttsm_tiles import check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M", [89, 96, 100, 108, 109])
def test_double_double_gram(handle, M):
    for K in (17, 300):
        check(handle, np.float64, "dd", M, M, K, gram=True)


@pytest.mark.parametrize("dt,M,N", [(np.complex128, 61, 393), (np.complex128, 218, 234), (np.float64, 246, 659),
                                    (np.float64, 36, 869), (np.complex64, 246, 659)])
def test_native(handle, dt, M, N):
    check(handle, dt, "native", M, N, 100)
    if dt == np.complex128:
        check(handle, dt, "native", M, N, 100, conj=True)


@pytest.mark.parametrize("dt,M", [(np.float32, 177), (np.float32, 216), (np.complex64, 89), (np.complex64, 108)])
def test_fp64_accumulation_of_fp32(handle, dt, M):
    K = 100
    rng = np.random.default_rng(M)
    A = common.uniform(rng, K * M, dt)
    Ad = torch.from_numpy(A).cuda()
    Cd = torch.zeros(M * M, dtype=Ad.dtype, device="cuda")
    handle.tsmttsm(M, M, K, Ad, M, 1.0, Ad, M, 0.0, Cd, M, acc="dd")
    wide = np.complex128 if dt == np.complex64 else np.float64
    X = A.astype(wide).reshape(K, M)
    exp = X.T @ X
    got = Cd.cpu().numpy().astype(wide).reshape(M, M).T
    # one rounding to FP32 (2^-24 of each part), sums of 100 products in FP64
    assert np.linalg.norm(got - exp) <= 2.0**-23 * np.linalg.norm(np.abs(X).T @ np.abs(X))
