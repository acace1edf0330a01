"""Split TSMTTSM, widths above 16: columns whose exponents rise at different stages (every stage, in
different warps, in the same stage), so that periods of one stage to a full one follow one another in
both TMEM sets; each compiled variant (folded or not, Gram block alone, among others, none; FP64 and
FP32); rows of a dense, a 16-byte aligned and an odd leading dimension; last stages cut short; columns
of zeros; exponents at the lower end of the range, where elements are subnormal.

The entries are integers below 2^20 (times a power of two), at most 2^14 of them in a sum with another
factor below 2^8: every digit product that the scheme drops is zero and every sum is below 2^53, so
the results are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (M, N, Gram)
SHAPES = [(17, 17, True), (32, 32, False), (32, 9, False), (33, 20, False), (64, 64, False), (64, 64, True),
          (100, 70, False), (100, 100, True)]


@pytest.mark.parametrize("dt,sa,sb", [(np.float64, 0, 0), (np.float64, -1070, 900), (np.float32, 0, 0)])
@pytest.mark.parametrize("M,N,gram", SHAPES)
def test_exponents_rise(handle, dt, sa, sb, M, N, gram):
    if gram and sa:
        pytest.skip("squares leave the range")
    for K in (1, 17, 50, 2500, 152 * 32 * 2 + 5):
        for pad in (0, 4, 3):
            rng = np.random.default_rng(M * 131 + N + K + pad)
            top = 5 if gram else 12
            r, c = np.arange(K)[:, None], np.arange(max(M, N) + pad)[None, :]
            grow = ((r // 16 + 3 * c) % 97) * top // 96
            A = rng.integers(-255, 256, (K, M + pad)) * (1 << grow[:, : M + pad])
            A[:, 0] = 0
            B = A if gram else rng.integers(-127, 128, (K, N + pad))
            exp = (B[:, :N].T @ A[:, :M]).astype(np.float64)
            assert np.abs(exp).max() < 2.0**53
            Ad = torch.from_numpy(np.ldexp(A.astype(np.float64), sa).astype(dt)).cuda()
            Bd = Ad if gram else torch.from_numpy(np.ldexp(B.astype(np.float64), sb).astype(dt)).cuda()
            Cd = torch.full((N, M), float("nan"), dtype=Ad.dtype, device="cuda")
            handle.tsmttsm(M, N, K, Ad, M + pad, 1.0, Bd, N + pad, 0.0, Cd, M, acc="split")
            assert np.array_equal(Cd.cpu().numpy(), np.ldexp(exp, sa + sb).astype(dt)), (K, pad)
