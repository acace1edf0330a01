"""SVQB of blocks with dependent columns: all equal, few distinct ones (random, or unit vectors), equal and
zero ones.  The null
vectors' eigenvalues agree to far below rounding (their gaps have no finite FP32 reciprocal).  All of Q is
finite, and the vectors of the nonzero eigenvalues (the last ones, eigenvalues ascend) are orthonormal to
what one pass leaves: 64 M u times the ratio of the largest to the smallest nonzero eigenvalue."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0**-53


@pytest.mark.parametrize("M", [8, 24, 32, 48, 64])
@pytest.mark.parametrize("kind", ["equal", "three", "half", "equal and zero", "unit"])
def test_dependent_columns(handle, M, kind):
    K = 3000
    for seed in range(20):
        rng = np.random.default_rng(1000 * seed + M)
        r = {"equal": 1, "three": 3, "half": M // 2, "equal and zero": 1, "unit": 5}[kind]
        if kind == "unit":
            at = rng.integers(0, r, M)
            r = len(np.unique(at))
            X = np.zeros((K, M))
            X[7 * at, np.arange(M)] = 1.0
        else:
            X = rng.standard_normal((K, r))[:, rng.permutation(np.arange(M) % r)]
        if kind == "equal and zero":
            X[:, rng.permutation(M)[: M // 2]] = 0.0
        Xd = torch.from_numpy(np.ascontiguousarray(X)).cuda()
        handle.svqb(K, M, Xd, M, gram_acc="native", orth_err=False)
        Q = Xd.cpu().numpy()
        assert np.isfinite(Q).all(), seed
        norm = np.linalg.norm(X, axis=0)
        lam = np.linalg.svd(X / np.where(norm > 0, norm, 1.0), compute_uv=False)[:r] ** 2
        Qr = Q[:, M - r:]
        assert np.linalg.norm(Qr.T @ Qr - np.eye(r)) <= 64 * M * U * lam[0] / lam[-1], seed
