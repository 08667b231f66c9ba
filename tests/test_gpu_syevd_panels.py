"""The eigensolver's panel reduction (one cooperative launch per 32 columns) at its edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 31, 32, 33, 34, 64, 65, 97, 400])
@pytest.mark.parametrize("kind", ["random", "graded", "diagonal", "banded"])
def test_panel_reduction_edges(handle, n, kind):
    # sizes around the 32-column panels and the 16 rows per CTA; columns with nothing below the
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
