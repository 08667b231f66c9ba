"""The eigensolver's reduction to tridiagonal form at its edges: in shared memory up to order 160, above in
panels of 32 columns (one cooperative launch each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("n", [2, 3, 16, 17, 33, 64, 97, 159, 160, 161, 192, 193, 194, 225, 400])
@pytest.mark.parametrize("kind", ["random", "graded", "diagonal", "banded"])
def test_panel_reduction_edges(handle, n, kind):
    # sizes around the two forms' border and the 32-column panels; columns with nothing below the
    # diagonal (no reflector) in the diagonal and banded matrices.  Backward stability: residual and
    # loss of orthogonality a small multiple of n 2^-53 of the norm
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    if kind == "graded":
        s = np.exp(-np.linspace(0, 30, n))
        A = A * s[:, None] * s[None, :]
    elif kind == "diagonal":
        A = np.diag(rng.standard_normal(n))
    elif kind == "banded":
        A = np.triu(np.tril(A, 1), -1)
        A[:, n // 2] = A[n // 2, :] = 0.0
    w, Z = handle.syevd(A)
    norm = max(np.linalg.norm(A, 2), 1e-300)
    assert np.linalg.norm(A @ Z - Z * w[None, :], 2) < 64 * n * 2.0 ** -53 * norm
    assert np.linalg.norm(Z.T @ Z - np.eye(n), 2) < 64 * n * 2.0 ** -53
    assert np.max(np.abs(w - np.linalg.eigvalsh(A))) < 64 * n * 2.0 ** -53 * norm
