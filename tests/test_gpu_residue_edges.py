"""Residue products (modgemm.cu) where their launches, memory and operands are at an edge: short launches one
after the other, descriptors rewritten in place, operands graded against each other, workspace caps at which
some of the optional buffers fit, expired waits."""
import numpy as np
import pytest

from oracle import rpa_oracle as O

pytestmark = pytest.mark.gpu


def test_short_launches_back_to_back(handle):
    # one tile per modulus, a single K chunk: CTA pairs start and end within microseconds, and the next
    # launch reuses their shared memory and accumulators.  Whole-number arithmetic: bitwise the same.
    x, _ = O.casimir_polder(1, 0.8)
    systems = [O.make_system(nq, 2, 64, nq, decay=30.0, lam0=0.8) for nq in (128, 200)]
    ref = [handle.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64") for s in systems]
    for it in range(400):
        s, r = systems[it & 1], ref[it & 1]
        assert np.array_equal(handle.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64"), r)


def _pi(n, k, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((k, n, 64)) * 0.05
    return X @ X.transpose(0, 2, 1)


def test_descriptors_rewritten_in_place(pkg):
    # tensor maps in descriptor arrays that every new shape fills again at the same address (log-det blocks,
    # split pass and SYRK of a batch): each call must see its own.  Fresh handles give the same bits.
    x, w = O.casimir_polder(2, 0.8)
    pis = [_pi(n, 2, n) for n in (1300, 1452, 1281)]
    sets = [[(s.R, s.eps_o, s.eps_v, x, w) for s in (O.make_system(nq, no, nv, nq, decay=30.0, lam0=0.8)
                                                     for nq, no, nv in shapes)]
            for shapes in ([(200, 4, 60), (1537, 3, 100)], [(1545, 4, 70), (190, 5, 66)], [(210, 3, 50), (180, 6, 30)])]
    ref_e, ref_b = [], []
    for pi, t in zip(pis, sets):
        with pkg.Handle(0) as h:
            h.set_autotune(False)
            ref_e.append(h.ec_from_pi(pi, np.ones(2))[1])
            ref_b.append(h.ec_batched(t, prec="split")[0])
    with pkg.Handle(0) as h:
        h.set_autotune(False)
        for it in range(12):
            i = (it * 2 + it // 3) % 3
            assert np.array_equal(h.ec_from_pi(pis[i], np.ones(2))[1], ref_e[i])
            assert np.array_equal(h.ec_batched(sets[i], prec="split")[0], ref_b[i])


@pytest.mark.parametrize("sd", [0.0, 2.0, 4.0])
def test_thc_vectors_from_graded_factors(handle, sd):
    # R(k, ai) = sum_g Z(g, k) Xa(g, a) Xi(g, i) does not change when grid points of Z are scaled by t(g) and
    # those of Xa by 1 / t(g) (log-normal t: sizes e^-3sd .. e^3sd and more), nor may its accuracy.  Powers of two
    # give the same bits; any t leaves the error below 16 units of 2^-53 of the sum of magnitudes, the rounding of
    # operands of even size (FP64 sums of 2500 terms stay within 2500).
    ng, nq, no, nv = 2500, 801, 12, 126
    Z, Xa, Xi, _, _ = O.make_thc_factors(ng, nq, no, nv, 5)
    rng = np.random.default_rng(17)
    t = np.exp(sd * rng.standard_normal(ng))
    two = np.exp2(np.rint(np.log2(t)))
    R = handle.thc_r(Z, Xa, Xi)
    assert np.array_equal(handle.thc_r(Z * two[:, None], Xa / two[:, None], Xi), R)
    Zs, Xs = Z * t[:, None], Xa / t[:, None]
    got = handle.thc_r(Zs, Xs, Xi)
    k = rng.integers(0, nq, 24)
    ai = rng.integers(0, no * nv, 40)
    a = Zs[:, k].astype(np.longdouble)
    b = (Xs[:, ai % nv].astype(np.longdouble) * Xi[:, ai // nv])
    ref, size = a.T @ b, np.abs(a).T @ np.abs(b)
    assert np.max(np.abs(got[np.ix_(k, ai)] - ref) / size) < 16 * 2.0 ** -53


def _graded_grad(handle, nq, no, nv, k, span):
    # rows of R from 1 down to e^-span, as pivoted Cholesky vectors fall off
    rng = np.random.default_rng(nq)
    nov = no * nv
    R = np.asfortranarray(rng.standard_normal((nq, nov)) * 0.05 * np.exp(-np.linspace(0, span, nq))[:, None])
    eo, ev = np.sort(rng.uniform(-1.0, -0.5, no)), np.sort(rng.uniform(0.1, 2.0, nv))
    x, w = O.casimir_polder(k, 0.8)
    _, dR, dO, dV = handle.ec_grad(R, eo, ev, x, w, prec="fp64")
    return R, eo, ev, x, w, dR


@pytest.mark.parametrize("nq, span", [(200, 0.0), (200, 20.0), (330, 30.0), (1300, 30.0)])
def test_gradient_rows_of_graded_vectors(handle, nq, span):
    # every row of dE/dR against its own size: (1 + Pi)^-1 - 1 = -X (1 + X^T X)^-1 X^T is graded as R is, and
    # so are the errors of a factorization of 1 + Pi and of its solves: nq roundings of 2^-53 per row, four-fold
    # for the two triangular factors and the two products.  Reference: the small side, 80-bit.
    R, eo, ev, x, w, dR = _graded_grad(handle, nq, 2, 64, 2, span)
    d = O.dai(eo, ev).astype(np.longdouble)
    Rl = R.astype(np.longdouble)
    ref = np.zeros(R.shape, np.longdouble)
    for u, f in zip(x, w):
        c = d / (d * d + np.longdouble(u) ** 2)
        X = Rl * np.sqrt(4.0 * c)[None, :]
        B = np.eye(R.shape[1], dtype=np.longdouble) + X.T @ X
        # (1 + X X^T)^-1 X = X B^-1; solve by Cholesky in 80 bits
        n = B.shape[0]
        L = np.zeros_like(B)
        for j in range(n):
            L[j:, j] = B[j:, j] - L[j:, :j] @ L[j, :j]
            L[j:, j] /= np.sqrt(L[j, j])
        Y = X.copy()  # rows times L^-T, then L^-1
        for j in range(n):
            Y[:, j] = (Y[:, j] - Y[:, :j] @ L[j, :j]) / L[j, j]
        for j in range(n - 1, -1, -1):
            Y[:, j] = (Y[:, j] - Y[:, j + 1:] @ L[j + 1:, j]) / L[j, j]
        # dE/dR = w / (2 pi) 2 alpha c ((1 + Pi)^-1 - 1) R: X column a is sqrt(4 c_a) R column a
        ref += f / (2 * np.pi) * 2.0 * np.sqrt(4.0 * c)[None, :] * (Y - X)
    err = np.linalg.norm((dR - ref).astype(float), axis=1) / np.linalg.norm(ref.astype(float), axis=1)
    assert np.max(err) < 16 * nq * 2.0 ** -53


def test_every_call_reports_an_expired_device_wait(pkg, monkeypatch):
    # the error word of the device as every check of it sees it: a call that does not look at it before it
    # answers would return RPA_OK with whatever an unfinished product left
    ng, nq, no, nv = 120, 30, 4, 10
    Z, Xa, Xi, eo, ev = O.make_thc_factors(ng, nq, no, nv, 9)
    s = O.make_system(40, no, nv, 3, decay=10.0, lam0=0.8)
    x, w = O.casimir_polder(4, 0.8)
    pi = O.pi_matrices(s.R, s.eps_o, s.eps_v, x)
    U, _ = np.linalg.qr(np.random.default_rng(2).standard_normal((no * nv, 8)))
    A = -0.1 * np.linspace(0.2, 1.0, 8)
    G = np.eye(40)[:, :20]
    calls = {
        "thc_r": lambda h: h.thc_r(Z, Xa, Xi),
        "ec_thc fp64": lambda h: h.ec_thc(Z, Xa, Xi, eo, ev, x, w, prec="fp64"),
        "ec_thc split": lambda h: h.ec_thc(Z, Xa, Xi, eo, ev, x, w, prec="split"),
        "project_basis": lambda h: h.project_basis(G, s.R),
        "piu_basis random": lambda h: h.piu_basis(s.R, s.eps_o, s.eps_v, 0.1, basis="random"),
        "piu_basis eigen": lambda h: h.piu_basis(s.R, s.eps_o, s.eps_v, 0.1, basis="eigen"),
        "dring_t2": lambda h: h.dring_t2(s.R, s.eps_o, s.eps_v, x, w),
        "mbpt3 fp64": lambda h: h.exchange_mbpt3(s.R, s.eps_o, s.eps_v, U, A, prec="fp64"),
        "mbpt3 split": lambda h: h.exchange_mbpt3(s.R, s.eps_o, s.eps_v, U, A, prec="split"),
        "sosex split": lambda h: h.exchange_sosex(s.R, no, nv, U, A, prec="split"),
        "jctc2024": lambda h: h.jctc2024(Z, Xi, Xa, U, A),
        "pi_u": lambda h: h.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64"),
        "ec fp64": lambda h: h.ec_rpa(s.R, s.eps_o, s.eps_v, x, w, prec="fp64"),
        "ec split": lambda h: h.ec_rpa(s.R, s.eps_o, s.eps_v, x, w, prec="split"),
        "ec_from_pi": lambda h: h.ec_from_pi(pi, w),
        "ec_grad": lambda h: h.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="fp64"),
        "ec_batched": lambda h: h.ec_batched([(s.R, s.eps_o, s.eps_v, x, w)] * 2, prec="split"),
    }
    with pkg.Handle(0) as h:
        for call in calls.values():
            call(h)  # each of them is sound as it stands
    monkeypatch.setenv("RPA_B200_SELFTEST_DEVICE_ERROR", "103")
    with pkg.Handle(0) as h:
        h.set_autotune(False)
        for name, call in calls.items():
            with pytest.raises(pkg.RPAError) as err:
                call(h)
            assert err.value.status == pkg.RPA_ERR_TIMEOUT, name


def _caps(pkg, call, monkeypatch, steps=24):
    """The call at caps from the least it runs with up to all it asks for: results, none of them refused."""
    def run(limit):
        with pkg.Handle(0) as h:
            h.set_autotune(False)
            h.set_workspace_limit(limit)
            try:
                out = call(h)
            except pkg.RPAError as e:
                assert e.status == pkg.RPA_ERR_OOM
                return None, h.workspace_bytes()[0]
            return out, h.workspace_bytes()[0]
    free, full = run(0)
    monkeypatch.setenv("RPA_B200_RESIDUES", "0")
    lo, hi = 0, full
    while hi - lo > max(full // 512, 4096):  # the least cap, everything on DMMA
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if run(mid)[0] is not None else (mid, hi)
    monkeypatch.setenv("RPA_B200_RESIDUES", "1")
    out = []
    for c in np.linspace(hi, full, steps):
        r, used = run(int(c))
        assert r is not None, "refused at a cap of %d bytes, %d suffice" % (c, hi)
        assert used <= c
        out.append(r)
    return free, out


@pytest.mark.parametrize("what", ["ec", "grad", "grad split", "t2", "batch"])
def test_optional_planes_never_cost_a_call_its_room(pkg, monkeypatch, what):
    # workspace caps at which some of the residue planes fit: what the call needs afterwards must still find
    # its room, whatever the planes took first.  The forms differ by their rounding only (tolerances as in
    # the tests of each form).
    monkeypatch.setenv("RPA_B200_RESIDUES", "1")
    nq, no, nv = (1540, 2, 70) if what == "batch" else (260, 4, 70)
    s = O.make_system(nq, no, nv, 9, decay=nq / 8.0, lam0=0.8)
    x, w = O.casimir_polder(3, 0.8)
    guess = np.random.default_rng(4).standard_normal((no * nv, 90))
    if what == "ec":
        call = lambda h: np.array([h.ec_rpa(s.R, s.eps_o, s.eps_v, x, w, prec="fp64")[0]])
    elif what == "grad":
        call = lambda h: h.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="fp64")[1]
    elif what == "grad split":
        call = lambda h: h.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="split")[1]
    elif what == "t2":
        call = lambda h: h.dring_t2(s.R, s.eps_o, s.eps_v, x, w, guess=guess, cutoff_thresh=1e-6)["A"]
    else:
        call = lambda h: h.ec_batched([(s.R, s.eps_o, s.eps_v, x, w)] * 2, prec="fp64")[0]
    free, out = _caps(pkg, call, monkeypatch, steps=10 if what == "batch" else 24)
    tol = 1e-12 if what != "t2" else 1e-9  # T2: eigenvalues of a Rayleigh-Ritz step, both forms in FP64
    for r in out:
        assert r.shape == free.shape
        assert np.max(np.abs(r - free)) < tol * np.max(np.abs(free))


def test_more_pairs_than_a_grid_dimension_holds(handle):
    # 128-wide chunks of ai beyond 65535: the FP64 pipe forms Pi (8.6 GB of vectors).  Sums of 8.4e6 products
    # of either sign, each rounded at 2^-53 of the partial sum, on both sides: 1e-11 of the norms is
    # 1e5 roundings, far above the sqrt(8.4e6) = 3e3 that independent ones leave.
    import torch
    no, nv, nq = 2049, 4096, 128
    assert no * nv > 65535 * 128
    g = torch.Generator(device="cuda").manual_seed(1)
    Rt = torch.randn((no * nv, nq), dtype=torch.float64, device="cuda", generator=g) * 1e-2
    eo, ev = np.sort(np.linspace(-2.0, -0.5, no)), np.sort(np.linspace(0.1, 3.0, nv))
    got = handle.pi_u(Rt.T, eo, ev, np.array([0.7]), prec="fp64")[0]
    d = torch.from_numpy((ev[None, :] - eo[:, None]).ravel()).cuda()
    c = 4.0 * d / (d * d + 0.49)
    ref = torch.zeros((nq, nq), dtype=torch.float64, device="cuda")
    for a in range(0, no * nv, 1 << 20):
        blk = Rt[a:a + (1 << 20)]
        ref += blk.T @ (blk * c[a:a + (1 << 20), None])
    n = torch.sqrt(torch.diagonal(ref))
    ref, n = ref.cpu().numpy(), n.cpu().numpy()
    assert np.max(np.abs(got - ref) / (n[:, None] * n[None, :])) < 1e-11


@pytest.mark.parametrize("scale", [1e140, 1e180, 1e280])
def test_log_det_of_very_large_pi(handle, scale):
    # squares of the off-diagonal entries leave the exponent range, the factorization does not: ln det is lost in
    # E(u) = ln det - Tr, which is -Tr to one rounding
    n = 130
    rng = np.random.default_rng(7)
    X = rng.standard_normal((2, n, n + 10)) / n
    pi = (X @ X.transpose(0, 2, 1)) * scale
    _, eu = handle.ec_from_pi(pi, np.ones(2))
    tr = np.trace(pi, axis1=1, axis2=2)
    assert np.all(np.abs(eu + tr) <= 2.0 ** -50 * tr)


@pytest.mark.parametrize("scale", [1.0, 1e-40, 1e-50, 1e30])
def test_random_basis_does_not_depend_on_the_size_of_pi(handle, scale):
    # CholeskyQR of Pi G: entries of its Gram matrix from 1e-200 to 1e120
    s = O.make_system(90, 4, 40, 3, decay=30.0, lam0=0.8)
    guess = np.random.default_rng(8).standard_normal((90, 90))
    ref, _, tr0 = handle.piu_basis(s.R, s.eps_o, s.eps_v, 0.1, target_error=0.0, basis="random", guess=guess)
    two = np.exp2(np.rint(np.log2(scale)))  # exact
    G, _, tr = handle.piu_basis(s.R * two, s.eps_o, s.eps_v, 0.1, target_error=0.0, basis="random", guess=guess)
    assert abs(tr - tr0 * two * two) <= 1e-14 * tr
    assert np.max(np.abs(np.abs(np.sum(G * ref, axis=0)) - 1.0)) < 1e-8


def test_eigensolvers_of_several_threads(pkg):
    # handles of their own, orders with other shared-memory sizes: the limit of a kernel is the process's
    import threading
    rng = np.random.default_rng(11)
    mats = [(lambda a: a + a.T)(rng.standard_normal((n, n))) for n in (170, 700, 301)]
    ref = [np.linalg.eigvalsh(a) for a in mats]
    failed = []

    def work(a, r):
        try:
            with pkg.Handle(0) as h:
                for _ in range(25):
                    w, _ = h.syevd(a)
                    assert np.max(np.abs(w - r)) < 64 * len(r) * 2.0 ** -53 * np.max(np.abs(r))
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=t) for t in zip(mats, ref)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.fixture
def forms(pkg, monkeypatch):
    """Two handles whose FP64 products run by residues (in blocks of 128 columns) and on DMMA, at any size."""
    hs = []
    for form in ("1", "0"):
        monkeypatch.setenv("RPA_B200_RESIDUES", form)
        monkeypatch.setenv("RPA_B200_GEMM64_BYTES", str(15 * (384 + 512) * 128))
        hs.append(pkg.Handle(0))
    yield hs
    for h in hs:
        h.close()


def _long_error(got, a, b):
    """Largest error of got = a^T b against 80 bits, relative to the norms of the two rows."""
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    n = np.sqrt(np.sum(al * al, axis=0))[:, None] * np.sqrt(np.sum(bl * bl, axis=0))[None, :]
    n[n == 0] = 1
    return float(np.max(np.abs(got - al.T @ bl) / n))


@pytest.mark.parametrize("nq, nvec, nov", [(1, 1, 1), (31, 7, 130), (128, 128, 256), (129, 127, 257), (300, 250, 391),
                                           (384, 384, 140)])
def test_projection_by_residues(forms, nq, nvec, nov):
    # R' = G^T R, both operands contiguous along the summed index; blocks of 128 columns of R'.  Operands are rounded
    # at 2^-58 of their norms and the result once at 2^-53: 4 2^-53 of the norms.  Columns of zeros, of
    # very different size, and one whose squares leave the exponent range.
    rng = np.random.default_rng(nq + nov)
    G, R = rng.standard_normal((nq, nvec)), np.asfortranarray(rng.standard_normal((nq, nov)))
    R *= np.exp(rng.uniform(-60, 60, nov))[None, :]
    R[:, ::17] = 0.0
    R[:, nov - 1] *= 1e170
    got = forms[0].project_basis(G, R)
    assert np.all(got[:, ::17][:, :-1] == 0.0)
    assert _long_error(got, G, R) < 4 * 2.0 ** -53
    assert _long_error(forms[1].project_basis(G, R), G, R) < max(nq, 4) * 2.0 ** -53


@pytest.mark.parametrize("ng, nq, no, nv", [(1, 1, 1, 1), (130, 33, 3, 50), (257, 200, 5, 61), (384, 129, 2, 64)])
def test_thc_vectors_by_residues(forms, ng, nq, no, nv):
    Z, Xa, Xi, _, _ = O.make_thc_factors(ng, nq, no, nv, 5)
    YX = (Xa.astype(np.longdouble)[:, None, :] * Xi.astype(np.longdouble)[:, :, None]).reshape(ng, no * nv)
    # the Khatri-Rao entries themselves are rounded at 2^-53
    assert _long_error(forms[0].thc_r(Z, Xa, Xi), Z, YX) < 6 * 2.0 ** -53
    assert _long_error(forms[1].thc_r(Z, Xa, Xi), Z, YX) < max(ng, 6) * 2.0 ** -53


def test_nan_in_an_operand_is_reported(forms, pkg):
    rng = np.random.default_rng(3)
    G, R = rng.standard_normal((140, 130)), np.asfortranarray(rng.standard_normal((140, 150)))
    for bad in (np.nan, np.inf):
        R[7, 149] = bad
        for h in forms:
            with pytest.raises(pkg.RPAError) as e:
                h.project_basis(G, R)
            assert e.value.status == pkg.RPA_ERR_NONFINITE


@pytest.mark.parametrize("nq, no, nv, nt", [(60, 3, 21, 30), (137, 4, 70, 129), (200, 5, 52, 140)])
def test_lyapunov_products_by_residues(forms, nq, no, nv, nt):
    # every operand order of the products, alpha = -1 with beta = 1, and a scale of the summed index (the orbital
    # energy differences): both forms solve the same equation to 1e-13 of its right-hand side
    s = O.make_system(nq, no, nv, nt, decay=nq / 6.0, lam0=0.8)
    U, _ = np.linalg.qr(np.random.default_rng(nt).standard_normal((no * nv, nt)))
    A = -np.exp(-np.linspace(1.5, 6.0, nt))
    out = [h.exchange_mbpt3(s.R, s.eps_o, s.eps_v, U, A, return_x=True) for h in forms]
    (e0, x0), (e1, x1) = out
    assert abs(e0 - e1) < 1e-11 * abs(e1)
    assert np.max(np.abs(x0 - x1)) < 1e-11 * np.max(np.abs(x1))


def test_amplitudes_and_basis_by_residues(forms):
    # T2 eigenvalues (rows contiguous times columns contiguous, both summed indices) and the random basis (an
    # operand times its own transpose): 1e-10 as in the tests of each against the oracle
    s = O.make_system(150, 4, 33, 2, decay=25.0, lam0=0.8)
    x, w = O.casimir_polder(5, 0.8)
    guess = np.random.default_rng(5).standard_normal((132, 120))
    t0, t1 = [h.dring_t2(s.R, s.eps_o, s.eps_v, x, w, guess=guess) for h in forms]
    assert t0["NT"] == t1["NT"]
    assert np.max(np.abs(t0["A"] - t1["A"])) < 1e-10 * np.max(np.abs(t1["A"]))
    assert np.max(np.abs(t0["EigRPA"] - t1["EigRPA"])) < 1e-10 * np.max(np.abs(t1["EigRPA"]))
    g = np.random.default_rng(6).standard_normal((90, 90))
    s = O.make_system(90, 4, 40, 3, decay=30.0, lam0=0.8)
    b0, b1 = [h.piu_basis(s.R, s.eps_o, s.eps_v, 0.1, target_error=0.0, basis="random", guess=g)[0] for h in forms]
    assert np.max(np.abs(np.abs(np.sum(b0 * b1, axis=0)) - 1.0)) < 1e-9


@pytest.mark.parametrize("nq, no, nv, k", [(1, 1, 1, 1), (5, 2, 9, 3), (127, 3, 40, 2), (100, 2, 30, 17)])
def test_small_pi_and_gradient_by_residues(forms, nq, no, nv, k):
    # below the sizes from which the residue forms are taken, both forms agree with the oracle
    s = O.make_system(nq, no, nv, nq + k, decay=nq / 4.0 + 1.0, lam0=0.8)
    x, w = O.casimir_polder(k, 0.8)
    ref = O.pi_matrices(s.R, s.eps_o, s.eps_v, x)
    gref = O.ec_grad(s.R, s.eps_o, s.eps_v, x, w)
    for h in forms:
        assert np.max(np.abs(h.pi_u(s.R, s.eps_o, s.eps_v, x, prec="fp64") - ref)) < 1e-13 * np.max(np.abs(ref))
        for a, b in zip(h.ec_grad(s.R, s.eps_o, s.eps_v, x, w, prec="fp64")[1:], gref):
            assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b))


def test_pivot_inverses(handle):
    # 1 / d and 1 / sqrt(d) of the diagonal blocks against the correctly rounded ones: a truncated series below
    # 2^-58.6 and two roundings, so within 2^-52 of the value; both sides of the switch to the library
    # functions, denormals, and pivots that are not positive
    rng = np.random.default_rng(13)
    m = np.concatenate([rng.uniform(1.0, 4.0, 60000), 1.0 + 2.0 ** -52 * np.arange(64), 4.0 - 2.0 ** -51 * np.arange(1, 64)])
    d = np.ldexp(m, rng.integers(-1020, 1021, m.size))
    edges = [x * (1.0 + 2.0 ** -52 * i) for x in (1e-290, 1e290) for i in range(-200, 200)]
    d = np.concatenate([d, m, edges, [1.0, 2.0, 0.5, 2.0 ** -1022, 2.0 ** 1022, 1.7e308]])
    inv, inv_sqrt = handle.selftest_pivots(d)
    dl = d.astype(np.longdouble)
    for got, ref in ((inv, 1 / dl), (inv_sqrt, 1 / np.sqrt(dl))):
        normal = ref > 2.3e-308  # 1 / d of the largest d is denormal
        err = np.abs(got - ref) / ref
        assert np.max(err[normal]) < 2.0 ** -52
        assert np.max(np.abs(got - ref)[~normal], initial=0.0) <= 2.0 ** -1074
    inv, inv_sqrt = handle.selftest_pivots(np.array([0.0, -1.0, -np.inf, np.nan]))
    assert np.all(inv == 1.0) and np.all(inv_sqrt == 1.0)


def test_energy_from_factors_in_pieces(pkg, monkeypatch):
    # pieces of 128 pairs that begin and end inside an occupied orbital: each piece's vectors as a residue
    # product, balanced over the orbitals it covers, against the vectors formed whole on the FP64 pipe
    ng, nq, no, nv = 300, 150, 5, 61
    Z, Xa, Xi, eo, ev = O.make_thc_factors(ng, nq, no, nv, 21)
    t = np.exp(3.0 * np.random.default_rng(22).standard_normal(ng))[:, None]
    x, w = O.casimir_polder(4, 0.8)
    monkeypatch.setenv("RPA_B200_RESIDUES", "0")
    with pkg.Handle(0) as h:
        R = h.thc_r(Z, Xa, Xi)
        ref = h.ec_rpa(R, eo, ev, x, w, prec="split")[0]
    monkeypatch.setenv("RPA_B200_RESIDUES", "1")
    monkeypatch.setenv("RPA_B200_THC_PIECE_BYTES", "1")
    monkeypatch.setenv("RPA_B200_GEMM64_BYTES", str(15 * (384 + 256) * 128))
    with pkg.Handle(0) as h:
        ec = h.ec_thc(Z * t, Xa / t, Xi, eo, ev, x, w, prec="split")[0]
    assert abs(ec - ref) < 1e-6  # split products in pieces against the whole, as in the pieces' own test
