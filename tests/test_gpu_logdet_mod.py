"""Log-det at the orders where its kernels change: the 64 x 64 diagonal factorization (every remainder of
its 8-column panels) and, from order 1280, trailing updates by residue products (256-column blocks,
128- and 256-row tiles; from 1536 in batches).

Tolerance: E(u) = ln det(1 + Pi) - Tr Pi, with 1 + Pi of eigenvalues in [1, 1 + lam]; the factorization's
backward error is below n 2^-53 per diagonal entry, so E(u) is off by at most n^2 2^-53 tr((1 + Pi)^-1) / n
<= n^2 2^-53 in the worst case and by about sqrt(n) n^(1/2) 2^-53 when the roundings are independent;
8 n 2^-53 is taken for both sides together.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_pi(n, k, seed):
    """k positive semidefinite matrices with largest eigenvalue about 0.8."""
    rng = np.random.default_rng(seed)
    out = np.empty((k, n, n))
    for i in range(k):
        X = rng.standard_normal((n, n + 8)) * np.exp(-np.arange(n) / (n / 6.0 + 1))[:, None]
        P = X @ X.T
        out[i] = P * (0.8 / np.linalg.norm(P, 2)) / (i + 1)
    return out


def reference(pi):
    w = [np.linalg.eigvalsh(p) for p in pi]
    return np.array([np.sum(np.log1p(x) - x) for x in w])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 40, 63, 64, 65, 71, 100, 127, 129])
def test_small_orders(handle, n):
    pi = random_pi(n, 2, n)
    _, eu = handle.ec_from_pi(pi, np.ones(2))
    assert np.max(np.abs(eu - reference(pi))) < 8 * max(n, 8) * 2.0 ** -53


@pytest.mark.parametrize("n", [1279, 1280, 1281, 1408, 1409, 1536, 1537])
def test_residue_updates(handle, n):
    pi = random_pi(n, 2, n)
    ref = reference(pi)
    for plan in ((128, 64), (256, 64), (512, 128)):
        handle.set_logdet_plan(n, *plan)
        _, eu = handle.ec_from_pi(pi, np.ones(2))
        assert np.max(np.abs(eu - ref)) < 8 * n * 2.0 ** -53


def test_residue_updates_without_room(pkg):
    # a workspace cap that holds Pi but not the planes: the updates stay on DMMA
    n = 1300
    pi = random_pi(n, 1, 5)
    with pkg.Handle(0) as h:
        h.set_autotune(False)
        h.set_workspace_limit(8 * n * n + (1 << 20))
        _, eu = h.ec_from_pi(pi, np.ones(1))
    assert np.max(np.abs(eu - reference(pi))) < 8 * n * 2.0 ** -53


def test_not_positive_definite_is_reported(handle, pkg):
    # a pivot that fails in the last block of a matrix whose updates run by residues
    n = 1300
    pi = random_pi(n, 1, 6)
    pi[0, n - 3, n - 3] = -1.5
    with pytest.raises(pkg.RPAError) as e:
        handle.ec_from_pi(pi, np.ones(1))
    assert e.value.status == pkg.RPA_ERR_NOT_SPD
    pi[0, n - 3, n - 3] = 0.1
    handle.ec_from_pi(pi, np.ones(1))


def test_batch_of_mixed_orders(handle):
    # one batched call over orders on both sides of the residue threshold, against single calls
    from oracle import rpa_oracle as O
    x, w = O.casimir_polder(3, 0.8)
    systems = []
    for nq, no, nv in [(300, 5, 61), (1537, 4, 100), (1601, 5, 90), (1540, 4, 120), (900, 4, 70), (1536, 3, 110)]:
        s = O.make_system(nq, no, nv, nq, decay=nq / 8.0, lam0=0.8)
        systems.append((s.R, s.eps_o, s.eps_v, x, w))
    ec, eu = handle.ec_batched(systems, prec="fp64")
    for t, e in zip(systems, eu):
        _, ref = handle.ec_rpa(*t, prec="fp64")
        # the batch forms Pi on the FP64 tensor pipe (nov additions per entry), the single call by residues
        assert np.max(np.abs(e - ref)) < 16 * t[0].shape[0] * 2.0 ** -53
