"""SVQB's eigensolver on the device: FP32 stage, FP64 refinement and the FP64 Jacobi behind it.

Widths around the smallest one that takes the FP32 stage (8), odd ones (a dummy player) and the
largest; spectra that the refinement alone finishes (well separated), that need FP64 sweeps (small
eigenvalues below FP32's rounding of the largest), an orthonormal block (every pair closer than its
coupling), blocks whose eigenvalues differ by 1e-9 only, and a zero column.

Bounds.  Well separated (condition 10 to 1e3): Q against the oracle's, column by column up to sign,
1e-9 relative, as the other SVQB tests.  All: the transform diagonalises the Gram, that is
||Q^T Q - I||_F <= 64 kappa(S) u with S the scaled Gram the solver sees (kappa(S) u is what one pass
loses by forming Q), and Q spans what X spans: ||X - Q (Q^T X)|| small by the same measure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import svqb as OS  # noqa: E402

U = 2.0 ** -53


def svqb(handle, X, K, M, gram="native"):
    Xd = torch.from_numpy(np.ascontiguousarray(X.ravel())).cuda()
    handle.svqb(K, M, Xd, M, gram_acc=gram, orth_err=False)
    return Xd.cpu().numpy().reshape(K, M)


def kappa(X):
    S = X.T @ X
    d = 1.0 / np.sqrt(np.diag(S))
    return np.linalg.cond(S * d[:, None] * d[None, :])


@pytest.mark.parametrize("M", [2, 3, 7, 8, 9, 16, 31, 40, 63, 64])
@pytest.mark.parametrize("cond", [10.0, 1e3])
def test_separated_spectra_match_the_oracle(handle, M, cond):
    K = 6001
    X = OS.make_x(K, M, cond, seed=M + 1)
    Q = svqb(handle, X, K, M)
    Qr = OS.svqb(X, K, M, "exact").reshape(K, M)
    s = np.sign(np.sum(Q * Qr, axis=0))
    assert np.linalg.norm(Q * s - Qr) <= 1e-9 * np.linalg.norm(Qr)
    assert np.linalg.norm(Q.T @ Q - np.eye(M)) <= 64 * kappa(X.reshape(K, M)) * U * M


@pytest.mark.parametrize("M", [8, 9, 33, 64])
@pytest.mark.parametrize("kind", ["ill", "orthonormal", "clustered"])
def test_spectra_that_fp32_cannot_separate(handle, M, kind):
    K = 4099
    rng = np.random.default_rng(M)
    if kind == "ill":
        X = OS.make_x(K, M, 1e6, seed=M).reshape(K, M)
    else:
        X = np.linalg.qr(rng.standard_normal((K, M)))[0]
        if kind == "clustered":
            X = X @ (np.eye(M) + 1e-9 * rng.standard_normal((M, M)))
    Q = svqb(handle, X, K, M)
    k = min(kappa(X), 1.0 / U)
    assert np.linalg.norm(Q.T @ Q - np.eye(M)) <= 64 * k * U * M
    if kind != "ill":
        assert np.linalg.norm(X - Q @ (Q.T @ X)) <= 64 * U * M * np.linalg.norm(X)


@pytest.mark.parametrize("M", [5, 12, 64])
def test_zero_column(handle, M):
    """A zero column has scale 0 and eigenvalue 0: its vector is scaled by 1e7.5 at most, and all
    other columns come out orthonormal."""
    K = 3000
    X = np.random.default_rng(M).standard_normal((K, M))
    X[:, M // 2] = 0.0
    Q = svqb(handle, X, K, M)
    assert np.all(np.isfinite(Q))
    S = Q.T @ Q
    assert np.linalg.norm(S[1:, 1:] - np.eye(M - 1)) <= 64 * 4 * U * M  # ascending: the zero comes first
    assert abs(S[0, 0]) <= 1e-10
