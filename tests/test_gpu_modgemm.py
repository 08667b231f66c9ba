"""Residue products on the int8 tensor cores (modgemm.cu): the FP64 form of Pi(u) and the adjoint's
back-contraction, at the edges of their 256 x 256 tiles (128 rows per CTA of a pair), 128-wide K chunks and
frequency groups.

Tolerances.  Operand rows are rounded to 2^-58 of their 2-norm, so an entry of Pi is off by at most
  0.5 sqrt(nov) 2^-57 2 ||X_Q|| ||X_P||  (rounding)  +  2^-53 |Pi_QP|  (one rounding of the result)
and by the error of the factors sqrt(alpha c), 4 2^-53 |Pi| each; 16 2^-53 ||X_Q|| ||X_P|| covers the
sum for nov <= 2^16.  The reference entries are 80-bit sums.
"""
import numpy as np
import pytest

from oracle import rpa_oracle as O

pytestmark = pytest.mark.gpu

# NQ, NOcc, NVirt, K: tile edges (128, 256, 512 rows), K chunks (128 ai), one and several frequency groups
SHAPES = [(128, 2, 64, 1), (129, 4, 33, 2), (255, 3, 43, 3), (256, 2, 64, 17), (257, 5, 77, 2), (385, 3, 64, 5),
          (513, 2, 65, 33), (640, 6, 128, 4)]


def norms(pi):
    d = np.sqrt(np.einsum("kii->ki", pi))
    return d[:, :, None] * d[:, None, :]


def pi_long(s, x, alpha=4.0):
    d = O.dai(s.eps_o, s.eps_v).astype(np.longdouble)
    R = s.R.astype(np.longdouble)
    out = np.empty((len(x), s.nq, s.nq))
    for k, u in enumerate(x):
        out[k] = ((R * (alpha * d / (d * d + np.longdouble(u) ** 2))[None, :]) @ R.T).astype(np.float64)
    return out


@pytest.mark.parametrize("nq,no,nv,k", SHAPES)
def test_pi_fp64_entries(handle, nq, no, nv, k):
    s = O.make_system(nq, no, nv, 7 * nq + k, decay=nq / 8.0, lam0=0.8)
    x, _ = O.casimir_polder(k, 0.8)
    keep = list(range(k)) if k <= 3 else [0, k // 2, k - 1]
    ref = pi_long(s, np.asarray(x)[keep])
    got = handle.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64")[keep]
    assert np.max(np.abs(got - ref) / norms(ref)) < 16 * 2.0 ** -53


def test_pi_fp64_scales_and_zero_rows(handle):
    # rows of very different size (each row has its own power of two) and rows of zeros
    s = O.make_system(200, 4, 60, 3, decay=25.0, lam0=0.8)
    scale = np.exp(np.linspace(-150, 30, 200))
    scale[[0, 77, 199]] = 0.0
    s.R = np.asfortranarray(s.R * scale[:, None])
    x, _ = O.casimir_polder(3, 0.8)
    ref = pi_long(s, x)
    got = handle.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64")
    n = norms(ref)
    live = n > 0
    assert np.all(got[~live] == 0.0)
    assert np.max(np.abs(got - ref)[live] / n[live]) < 16 * 2.0 ** -53


def test_pi_fp64_padded_columns_and_small_workspace(handle, pkg):
    # a leading dimension larger than NQ (the padding is NaN), and a workspace cap with no room for
    # the residue planes: the DMMA form answers, within the two forms' rounding
    import torch
    s = O.make_system(300, 4, 70, 9, decay=40.0, lam0=0.8)
    x, w = O.casimir_polder(4, 0.8)
    big = np.full((313, s.R.shape[1]), np.nan)
    big[:300] = s.R
    R = torch.from_numpy(np.ascontiguousarray(big.T)).cuda().T[:300]
    ref = pi_long(s, x)
    got = handle.pi_u(R, s.eps_o, s.eps_v, x, prec="fp64")
    assert np.max(np.abs(got - ref) / norms(ref)) < 16 * 2.0 ** -53
    with pkg.Handle(0) as h:
        h.set_workspace_limit(4 * 300 * 300 * 8 + 300 * 280 * 8 + (1 << 20))
        capped = h.pi_u(R, s.eps_o, s.eps_v, x, prec="fp64")
    assert np.max(np.abs(capped - ref) / norms(ref)) < 280 * 2.0 ** -53  # 280 sequential FP64 additions


@pytest.mark.parametrize("nq,no,nv,k", [(127, 2, 64, 2), (128, 2, 64, 2), (193, 4, 33, 3), (257, 5, 77, 17), (321, 3, 64, 5),
                                        (1100, 8, 32, 35)])
def test_gradient_fp64(handle, nq, no, nv, k):
    # dE/dR and dE/de against the FP64 oracle: 1 + Pi has eigenvalues in [1, 1.8], so inverse and
    # products lose a few roundings of sqrt(NQ) terms; 1e-13 of the largest entry bounds both sides
    s = O.make_system(nq, no, nv, nq + k, decay=nq / 8.0, lam0=0.8)
    x, w = O.casimir_polder(k, 0.8)
    ref = O.ec_grad(s.R, s.eps_o, s.eps_v, x, w)
    ec, dR, dO, dV = handle.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="fp64")
    for a, b in zip((dR, dO, dV), ref):
        assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b))


def test_gradient_without_room_for_planes(pkg):
    # a cap that holds the triangular solves' buffers but not the residue planes
    s = O.make_system(160, 4, 60, 5, decay=20.0, lam0=0.8)
    x, w = O.casimir_polder(3, 0.8)
    ref = O.ec_grad(s.R, s.eps_o, s.eps_v, x, w)
    with pkg.Handle(0) as h:
        h.set_workspace_limit(3 << 20)
        _, dR, dO, dV = h.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="fp64")
    for a, b in zip((dR, dO, dV), ref):
        assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b))
