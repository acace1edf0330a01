"""Split TSMTTSM, widths up to 16: sums over several periods before the digit pairs are sorted by level
(more periods than are summed at a time; fewer; one), exponents that rise now and then or every round,
rounds read from global memory, last rounds cut short, columns of zeros, elements that are subnormal.

The entries are integers below 2^20 (times a power of two): every digit product that the scheme drops
is zero and every sum is below 2^53, so the results are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LONG = 152 * 1024 * 17 + 9  # above 15 periods of 1024 rows in every block

# (M, N, Gram, K)
CASES = [(1, 1, False, LONG), (2, 3, False, LONG), (4, 4, True, LONG)] + [
    (M, N, g, K) for (M, N, g) in ((8, 8, False), (7, 5, False), (16, 16, False), (16, 2, False), (2, 16, False),
                                   (8, 8, True), (16, 16, True), (13, 13, True)) for K in (1, 130, 5000, 152 * 1024 + 7)]


@pytest.mark.parametrize("dt,sa,sb", [(np.float64, 0, 0), (np.float64, -1070, 900), (np.float32, 0, 0)])
@pytest.mark.parametrize("M,N,gram,K", CASES)
def test_periods(handle, dt, sa, sb, M, N, gram, K):
    if gram and sa:
        pytest.skip("squares leave the range")
    for step in (100, 20000):  # rows between two rises of an exponent, about
        for pad in (0, 1) if K < LONG else (0,):
            rng = np.random.default_rng(M * 17 + N + K + pad)
            top = 5 if gram else 12
            r, c = np.arange(K)[:, None], np.arange(max(M, N) + pad)[None, :]
            grow = ((r // step + 3 * c) % 97) * top // 96
            A = rng.integers(-255, 256, (K, M + pad)) * (1 << grow[:, : M + pad])
            if M > 1:
                A[:, 0] = 0
            B = A if gram else rng.integers(-127, 128, (K, N + pad))
            exp = (B[:, :N].T @ A[:, :M]).astype(np.float64)
            assert np.abs(exp).max() < 2.0**53
            Ad = torch.from_numpy(np.ldexp(A.astype(np.float64), sa).astype(dt)).cuda()
            Bd = Ad if gram else torch.from_numpy(np.ldexp(B.astype(np.float64), sb).astype(dt)).cuda()
            Cd = torch.full((N, M), float("nan"), dtype=Ad.dtype, device="cuda")
            handle.tsmttsm(M, N, K, Ad, M + pad, 1.0, Bd, N + pad, 0.0, Cd, M, acc="split")
            assert np.array_equal(Cd.cpu().numpy(), np.ldexp(exp, sa + sb).astype(dt)), (step, pad)
