"""SVQB of a block that holds NaN or an infinity: the eigenvalues still rank as a permutation (no index is
left unset), the call returns, every vector is NaN, and the handle goes on working."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M", [2, 5, 7, 8, 9, 31, 64])
@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_every_vector_is_nan(handle, dt, M, bad):
    K = 3000
    rng = np.random.default_rng(M)
    X = rng.standard_normal((K, M)).astype(dt)
    for cols in ([M // 2], range(M)):
        Y = X.copy()
        for c in cols:
            Y[(7 * c + 5) % K, c] = bad
        Yd = torch.from_numpy(Y).cuda()
        handle.svqb(K, M, Yd, M, gram_acc="native", orth_err=False)
        assert np.isnan(Yd.cpu().numpy()).all()
    Xd = torch.from_numpy(X).cuda()
    handle.svqb(K, M, Xd, M, gram_acc="native", orth_err=False)
    Q = Xd.cpu().numpy()
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(M)) <= 1e-11
