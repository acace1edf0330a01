"""A product captured into a CUDA graph after a larger one ran on the same stream allocates nothing, whatever tile its
widths take, and the graph gives the eager call's bits."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt,acc,big,smaller", [
    (np.complex128, "native", 48, [(43, 45), (45, 43), (48, 1), (17, 33)]),
    (np.float32, "dd", 32, [(25, 29), (29, 25), (31, 31), (8, 8)]),
    (np.complex64, "dd", 48, [(43, 45), (40, 48)]), (np.float64, "native", 64, [(63, 61), (33, 64), (20, 20)])])
def test_smaller_widths(dt, acc, big, smaller):
    from skinny_matmul_gb300 import Handle
    h, s = Handle(0), torch.cuda.Stream()
    K = 100003
    rng = np.random.default_rng(big)
    A = torch.from_numpy(common.uniform(rng, K * big, dt)).cuda()
    B = torch.from_numpy(common.uniform(rng, K * big, dt)).cuda()

    def run(M, N, C):
        h.tsmttsm(M, N, K, A, M, 1.0, B, N, 0.0, C, M, acc=acc, stream=s.cuda_stream)
    torch.cuda.synchronize()
    run(big, big, torch.zeros(big * big, dtype=A.dtype, device="cuda"))
    torch.cuda.synchronize()
    for M, N in smaller:
        C = torch.zeros(M * N, dtype=A.dtype, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            run(M, N, C)
        g.replay()
        torch.cuda.synchronize()
        E = torch.zeros_like(C)
        torch.cuda.synchronize()
        run(M, N, E)
        torch.cuda.synchronize()
        assert torch.equal(C, E) and bool(torch.any(C != 0))
    h.close()
