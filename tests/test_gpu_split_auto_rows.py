"""AUTO accumulation of FP64 TSMTTSM with a width below 8 and the other above 16: the split kernel for dense operands and
for columns of a wide block, the CUDA-core kernel for rows with a few more columns; bit for bit."""
import numpy as np
import pytest

import common
from skinny_matmul_gb300 import api

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,N", [(4, 32), (6, 48), (64, 4)])
@pytest.mark.parametrize("pad,first,route", [(0, 0, "split"), (1, 0, "native"), (2, 0, "native"), (0, 1, "split"), (150, 1, "split")])
def test_route(M, N, pad, first, route):
    handle = api.Handle(0)  # of its own: an autotuned key overrides the rule
    K = (3 << 22) // (M * N) + 7
    rng = np.random.default_rng(M + N + pad)
    A = torch.from_numpy(common.uniform(rng, K * (M + pad) + first, np.float64)).cuda()
    B = torch.from_numpy(common.uniform(rng, K * (N + pad) + first, np.float64)).cuda()
    out = []
    for acc in ("auto", "split", "native"):
        C = torch.zeros(M * N, dtype=A.dtype, device="cuda")
        handle.tsmttsm(M, N, K, A.data_ptr() + 8 * first, M + pad, 1.0, B.data_ptr() + 8 * first, N + pad, 0.0, C, M,
                       acc=acc, dtype=1)
        out.append(C.cpu().numpy())
    assert np.array_equal(out[0], out[1 if route == "split" else 2])
    assert not np.array_equal(out[1], out[2])
