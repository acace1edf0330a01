"""The autotuner may find that the untuned launch is the fastest: 1 x 1 and 2 x 2 FP32 products of many rows stream with
all CTAs that fit an SM (29 us at 2^24 rows; 48 with two, the most that the other candidates ask for)."""
import json

import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,K", [(1, 1 << 24), (2, 1 << 23)])
def test_untuned_launch_is_a_candidate(M, K):
    from skinny_matmul_gb300 import Handle
    h = Handle(0)
    h.autotune("tsmttsm", "float32", M, M, K, acc="native")
    (e,) = json.loads(h.tune_export())["entries"]
    assert (e["blocks_per_sm"], e["rows_per_tile"]) == (0, 0)
    k = 5003
    rng = np.random.default_rng(M)
    A, B = common.uniform(rng, k * M, np.float32), common.uniform(rng, k * M, np.float32)
    C = torch.zeros(M * M, dtype=torch.float32, device="cuda")
    h.tsmttsm(M, M, k, torch.from_numpy(A).cuda(), M, 1.0, torch.from_numpy(B).cuda(), M, 0.0, C, M)
    exp, den = common.tsmttsm_expected(M, M, k, A.astype(np.float64), M, B.astype(np.float64), M, np.zeros(M * M), M, 1.0, 0.0)
    assert common.normwise(C.cpu().numpy(), exp, den) <= common.tol(np.float32, k)
    h.close()
