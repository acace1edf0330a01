"""AUTO accumulation of FP64 / complex FP64 TSMTTSM: on either side of each line of the selection rule the
result is bit for bit that of the kernel that the rule names."""
import numpy as np
import pytest

import common
from skinny_matmul_gb300 import api

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

S, N_ = "split", "native"


@pytest.mark.parametrize("dt,M,N,K,route", [
    (np.float64, 8, 8, 1 << 16, S), (np.float64, 8, 8, (1 << 16) - 1, N_), (np.float64, 16, 16, 4096, N_),
    (np.float64, 32, 32, 4096, S), (np.float64, 64, 64, 4095, N_), (np.float64, 4, 8, 3 << 17, S),
    (np.float64, 4, 8, (3 << 17) - 1, N_), (np.float64, 4, 4, 1 << 20, N_), (np.float64, 3, 16, 1 << 19, N_),
    (np.float64, 4, 64, 1 << 16, S), (np.float64, 4, 63, 1 << 16, N_), (np.float64, 4, 32, 3 << 15, S),
    (np.float64, 4, 31, 1 << 17, N_), (np.complex128, 16, 16, 8192, N_), (np.complex128, 16, 16, 8193, S),
    (np.complex128, 8, 8, 1 << 14, S), (np.complex128, 8, 8, (1 << 14) - 1, N_), (np.complex128, 4, 2, 3 << 17, S)])
def test_route(dt, M, N, K, route):
    handle = api.Handle(0)  # of its own: an autotuned key overrides the rule
    rng = np.random.default_rng(M + N + K)
    A = torch.from_numpy(common.uniform(rng, K * M, dt)).cuda()
    B = torch.from_numpy(common.uniform(rng, K * N, dt)).cuda()
    out = []
    for acc in ("auto", S, N_):
        C = torch.zeros(M * N, dtype=A.dtype, device="cuda")
        handle.tsmttsm(M, N, K, A, M, 1.0, B, N, 0.0, C, M, acc=acc)
        out.append(C.cpu().numpy())
    assert np.array_equal(out[0], out[1 if route == S else 2])
    assert not np.array_equal(out[1], out[2])
