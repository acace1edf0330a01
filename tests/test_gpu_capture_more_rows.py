"""AUTO products captured into a CUDA graph after one of the same widths with fewer rows (4096 at least) ran on the
stream: the rule may take the split kernel for the captured one and not for the other, and nothing is allocated."""
import numpy as np
import pytest

import common

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt,M,N", [(np.float64, 24, 24), (np.float64, 32, 8), (np.complex128, 16, 16),
                                    (np.complex128, 13, 7), (np.float64, 17, 16)])
@pytest.mark.parametrize("gram", [False, True])
def test_more_rows(dt, M, N, gram):
    from skinny_matmul_gb300 import Handle
    h, s = Handle(0), torch.cuda.Stream()
    N = M if gram else N
    K = 60001
    rng = np.random.default_rng(M)
    A = torch.from_numpy(common.uniform(rng, K * M, dt)).cuda()
    B = A if gram else torch.from_numpy(common.uniform(rng, K * N, dt)).cuda()
    out = [torch.zeros(M * N, dtype=A.dtype, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()

    def run(k, C, acc="auto"):
        h.tsmttsm(M, N, k, A, M, 1.0, B, N, 0.0, C, M, acc=acc, stream=s.cuda_stream)
    run(4096, out[0])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        run(K, out[1])
    g.replay()
    torch.cuda.synchronize()
    run(K, out[2], "split")
    torch.cuda.synchronize()
    assert torch.equal(out[1], out[2])
    h.close()
