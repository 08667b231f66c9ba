"""The measured cases: what a user of the library has it compute, through the public entry points.

One handle serves every call of the process, as a program that works through many systems keeps one.
Cholesky vectors, THC factors and amplitudes are on the GPU before a call (the producers leave them
there); orbital energies, grids and eigenvalues are short host arrays.  Inputs have the distributions
of the benchmark's synthetic systems: Gaussian R(Q, ai) whose rows decay with Q, scaled so that the
largest eigenvalue of Pi(0) is 0.8, occupied energies uniform, virtual energies log-uniform.

Kinds of case (`"kind"`):
  energy    E_c of one system: Handle.ec_rpa
  pi        Pi(u) itself, then E_c from it: Handle.pi_u and Handle.ec_from_pi (codes that keep Pi)
  batch     E_c of many fragments of uneven size in one call: Handle.ec_batched
  grad      E_c and dE_c/d(R, energies): Handle.ec_grad
  autograd  a training or optimisation step through torch: rpa_energy forward and backward
  mbe       the many-body driver with exchange: Handle.mbe_beyond_rpa (grid, RPA, ring T2, SOSEX)
  exchange  SOSEX and MBPT3 exchange energies of given amplitudes
  thc       E_c from tensor-hypercontraction factors: Handle.ec_thc
  pno       the particle-hole corrections with pair-natural orbitals: Handle.jctc2024
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
_HANDLE = None


def _package():
    """The package (a hyphenated folder), imported as beyond_rpa_b200."""
    name = "beyond_rpa_b200"
    if name not in sys.modules:
        folder = ROOT / "beyond-rpa_b200"
        spec = importlib.util.spec_from_file_location(name, folder / "__init__.py",
                                                      submodule_search_locations=[str(folder)])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _handle():
    global _HANDLE
    if _HANDLE is None:
        _HANDLE = _package().Handle(0)
    return _HANDLE


def listed():
    return [
        # a water dimer in a double-zeta basis: the smallest system, where launches and latency count
        dict(name="dimer", kind="energy", nq=400, no=8, nv=72, k=12, prec="split"),
        # an odd-sized medium molecule
        dict(name="medium_odd", kind="energy", nq=1387, no=29, nv=331, k=10, prec="split"),
        # the benchmark's single system
        dict(name="single_4096", kind="energy", nq=4096, no=64, nv=1024, k=16, prec="split"),
        # the FP64 form: reference energies, validation of the split form
        dict(name="single_2048_fp64", kind="energy", nq=2048, no=32, nv=512, k=16, prec="fp64"),
        # Pi(u) kept by the caller, FP64, odd sizes
        dict(name="pi_fp64_odd", kind="pi", nq=777, no=21, nv=203, k=9, prec="fp64"),
        # a share of a many-body expansion: dimers and trimers of uneven size, 8 to 16 points each
        dict(name="fragments_24", kind="batch", n=24, lo=16, hi=48, prec="split"),
        # the gradient at the benchmark's adjoint shape
        dict(name="gradient_2560", kind="grad", nq=2560, no=48, nv=640, k=16, prec="split"),
        # a small differentiable energy inside a torch program
        dict(name="autograd_641", kind="autograd", nq=641, no=16, nv=161, k=12, prec="split"),
        # interaction energy of a dimer beyond RPA: three subsystems, ring amplitudes and SOSEX of each
        dict(name="mbe_dimer", kind="mbe", nq=768, no=24, nv=192, k=12, prec="split"),
        # both exchange energies of one set of amplitudes
        dict(name="exchange_1536", kind="exchange", nq=1536, no=40, nv=400, nt=900, prec="split"),
        # the energy from THC factors
        dict(name="thc_2048", kind="thc", ng=4096, nq=2048, no=32, nv=512, k=11, prec="split"),
        # PNO corrections of a small molecule
        dict(name="pno_256", kind="pno", ng=1024, nq=256, no=16, nv=128, nt=300),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "energy", "pi", "batch", "grad", "autograd", "mbe", "exchange", "thc", "pno"])
    if kind == "energy":
        prec = rng.choice(["split", "split", "fp64"])
        top = 4096 if prec == "split" else 2048
        return dict(kind=kind, nq=_between(rng, 120, top), no=_between(rng, 4, top // 64),
                    nv=_between(rng, 30, top // 4), k=rng.randint(6, 16), prec=prec)
    if kind == "pi":
        return dict(kind=kind, nq=_between(rng, 120, 1500), no=_between(rng, 4, 30), nv=_between(rng, 30, 330),
                    k=rng.randint(4, 12), prec=rng.choice(["split", "fp64"]))
    if kind == "batch":
        lo = rng.randint(6, 24)
        return dict(kind=kind, n=rng.randint(6, 24), lo=lo, hi=lo + rng.randint(6, 24), prec="split")
    if kind == "grad":
        return dict(kind=kind, nq=_between(rng, 150, 2000), no=_between(rng, 5, 40), nv=_between(rng, 40, 500),
                    k=rng.randint(6, 16), prec=rng.choice(["split", "fp64"]))
    if kind == "autograd":
        return dict(kind=kind, nq=_between(rng, 120, 1200), no=_between(rng, 4, 24), nv=_between(rng, 40, 300),
                    k=rng.randint(6, 14), prec="split")
    if kind == "mbe":
        return dict(kind=kind, nq=_between(rng, 200, 760), no=2 * rng.randint(4, 12), nv=2 * rng.randint(30, 96),
                    k=rng.randint(8, 12), prec=rng.choice(["split", "fp64"]))
    if kind == "exchange":
        return dict(kind=kind, nq=_between(rng, 200, 1500), no=_between(rng, 6, 40), nv=_between(rng, 50, 400),
                    nt=_between(rng, 150, 900), prec=rng.choice(["split", "split", "fp64"]))
    if kind == "thc":
        nq = _between(rng, 200, 2000)
        return dict(kind=kind, ng=2 * nq + rng.randint(0, 60), nq=nq, no=_between(rng, 6, 32),
                    nv=_between(rng, 50, 512), k=rng.randint(6, 11), prec="split")
    return dict(kind=kind, ng=_between(rng, 300, 1000), nq=_between(rng, 80, 256), no=rng.randint(6, 16),
                nv=_between(rng, 48, 128), nt=_between(rng, 80, 300))


# ------------------------------------------------------------------------------------------ inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, rows, cols):
    """Column-major (rows, cols) standard normal matrix."""
    return torch.randn((cols, rows), generator=g, device="cuda", dtype=torch.float64).T


def _energies(no, nv, seed):
    rng = np.random.default_rng(seed)
    eo = np.sort(rng.uniform(-1.3, -0.4, no))
    ev = np.sort(np.exp(rng.uniform(math.log(0.03), math.log(4.0), nv)))
    return eo, ev


def _gaps(eo, ev):
    """D(ai) = e_a - e_i with ai = a + NVirt * i."""
    return torch.from_numpy((ev[:, None] - eo[None, :]).reshape(-1, order="F")).cuda()


def _vectors(nq, eo, ev, seed):
    """R(Q, ai), column-major on the GPU, with lambda_max(Pi(0)) = 0.8 (power iteration)."""
    g = _generator(seed)
    R = _normal(g, nq, len(eo) * len(ev))
    R.mul_(torch.exp(-torch.arange(nq, device="cuda", dtype=torch.float64) / (nq / 8.0))[:, None])
    d = _gaps(eo, ev)
    v = torch.randn(nq, generator=g, device="cuda", dtype=torch.float64)
    for _ in range(20):
        w = 4.0 * (R @ ((R.T @ v) / d))
        lam = torch.linalg.norm(w)
        v = w / lam
    R.mul_(torch.sqrt(0.8 / lam))
    return R


def _system(nq, no, nv, k, seed):
    eo, ev = _energies(no, nv, seed)
    x, w = _package().freq_grid(np.concatenate([eo, ev]), no, nv, nfixed=k)
    return _vectors(nq, eo, ev, seed + 1), eo, ev, x, w


def _fragments(case, seed):
    """(NQ, NOcc, NVirt, K) of each fragment: the molecules are the same for every seed of a case."""
    rng = np.random.default_rng(1000 * case["n"] + 10 * case["lo"] + case["hi"])
    out = []
    for _ in range(case["n"]):
        no = int(rng.integers(case["lo"], case["hi"] + 1))
        nv = int(round(rng.uniform(8.0, 12.0) * no))
        out.append((4 * (no + nv), no, nv, int(rng.choice([8, 12, 16]))))
    return out


def _subsystems(case):
    """(NQ, NOcc, NVirt) of a dimer and its two monomers."""
    no, nv, nq = case["no"], case["nv"], case["nq"]
    return [(nq, no, nv), (nq // 2, no // 2, nv // 2), (nq // 2 + 8, no // 2, nv // 2)]


def _amplitudes(nov, nt, seed):
    """T2 = U diag(A) U^T: orthonormal columns (as the ring solver returns them), A < 0 decaying."""
    U = torch.linalg.qr(_normal(_generator(seed), nov, nt))[0]
    return U.T.contiguous().T, -0.2 * np.exp(-np.arange(nt) / (nt / 5.0))


def _thc(case, seed):
    ng, nq, no, nv = case["ng"], case["nq"], case["no"], case["nv"]
    g = _generator(seed)
    Z = _normal(g, ng, nq)
    Z.mul_((0.3 / math.sqrt(no * nv)) * torch.exp(-torch.arange(nq, device="cuda", dtype=torch.float64) / (nq / 8.0))[None, :])
    Xa = _normal(g, ng, nv).mul_(ng ** -0.25)
    Xi = _normal(g, ng, no).mul_(ng ** -0.25)
    return Z, Xa, Xi


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case, handle=_handle())
    seed = 7919 * int(seed) + 11
    if kind in ("energy", "pi", "grad", "autograd"):
        s["sys"] = _system(case["nq"], case["no"], case["nv"], case["k"], seed)
        R, eo, ev, x, w = s["sys"]
        if kind == "pi":
            s["out"] = torch.empty((case["k"], case["nq"], case["nq"]), dtype=torch.float64, device="cuda")
        elif kind == "grad":
            s["eo"], s["ev"] = torch.from_numpy(eo).cuda(), torch.from_numpy(ev).cuda()
            s["out"] = (torch.empty_like(R.T).T, torch.empty_like(s["eo"]), torch.empty_like(s["ev"]))
        elif kind == "autograd":
            from beyond_rpa_b200 import autograd
            s["energy"] = autograd.rpa_energy
            s["leaves"] = [R.requires_grad_(True), torch.from_numpy(eo).cuda().requires_grad_(True),
                           torch.from_numpy(ev).cuda().requires_grad_(True)]
            s["grid"] = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    elif kind == "batch":
        s["systems"] = [_system(nq, no, nv, k, seed + 17 * i)
                        for i, (nq, no, nv, k) in enumerate(_fragments(case, seed))]
    elif kind == "mbe":
        s["subsystems"] = []
        for i, (nq, no, nv) in enumerate(_subsystems(case)):
            eo, ev = _energies(no, nv, seed + 17 * i)
            s["subsystems"].append((_vectors(nq, eo, ev, seed + 17 * i + 1), eo, ev))
    elif kind == "exchange":
        eo, ev = _energies(case["no"], case["nv"], seed)
        s["eo"], s["ev"] = eo, ev
        s["R"] = _vectors(case["nq"], eo, ev, seed + 1)
        s["U"], s["A"] = _amplitudes(case["no"] * case["nv"], case["nt"], seed + 2)
    elif kind == "thc":
        s["eo"], s["ev"] = _energies(case["no"], case["nv"], seed)
        s["grid"] = _package().freq_grid(np.concatenate([s["eo"], s["ev"]]), case["no"], case["nv"],
                                         nfixed=case["k"])
        s["factors"] = _thc(case, seed + 1)
    else:
        s["factors"] = _thc(case, seed + 1)
        s["U"], s["A"] = _amplitudes(case["no"] * case["nv"], case["nt"], seed + 2)
    torch.cuda.synchronize()  # the handle computes on its own stream: its inputs are finished before a call
    return s


# ------------------------------------------------------------------------------------------ the pass

def run(s):
    h, kind = s["handle"], s["kind"]
    if kind == "energy":
        R, eo, ev, x, w = s["sys"]
        ec, eu = h.ec_rpa(R, eo, ev, x, w, prec=s["prec"])
        return {"ec": ec, "eu": eu}
    if kind == "pi":
        R, eo, ev, x, w = s["sys"]
        pi = h.pi_u(R, eo, ev, x, prec=s["prec"], out=s["out"])
        ec, eu = h.ec_from_pi(pi, w)
        return {"pi": pi, "ec": ec, "eu": eu}
    if kind == "batch":
        ec, eu = h.ec_batched(s["systems"], prec=s["prec"])
        return {"ec": ec, "eu": eu}
    if kind == "grad":
        R, _, _, x, w = s["sys"]
        ec, dR, dO, dV = h.ec_grad(R, s["eo"], s["ev"], x, w, prec=s["prec"], out=s["out"])
        return {"ec": ec, "dR": dR, "dO": dO, "dV": dV}
    if kind == "autograd":
        for t in s["leaves"]:
            t.grad = None
        e = s["energy"](*s["leaves"], *s["grid"], h, prec=s["prec"])
        e.backward()
        return {"ec": e.detach(), "grads": [t.grad for t in s["leaves"]]}
    if kind == "mbe":
        r = h.mbe_beyond_rpa(s["subsystems"], 2, prec=s["prec"], nfixed=s["k"], cutoff_thresh=1e-4)
        # the interaction energies eint and ex_int are left out: plain differences of ec and of ex, whose
        # relative error is set by how much cancels for the seed
        return {k: r[k] for k in ("freqs", "weights", "ec", "ex", "eig_rpa", "nt", "common_thresh")}
    if kind == "exchange":
        no, nv = s["no"], s["nv"]
        return {"sosex": h.exchange_sosex(s["R"], no, nv, s["U"], s["A"], prec=s["prec"]),
                "mbpt3": h.exchange_mbpt3(s["R"], s["eo"], s["ev"], s["U"], s["A"], prec=s["prec"])}
    if kind == "thc":
        Z, Xa, Xi = s["factors"]
        ec, eu = h.ec_thc(Z, Xa, Xi, s["eo"], s["ev"], *s["grid"], prec=s["prec"])
        return {"ec": ec, "eu": eu}
    Z, Xa, Xi = s["factors"]
    energies, counts = h.jctc2024(Z, Xi, Xa, s["U"], s["A"], cutoff_pno=1e-5)
    return {"energies": np.array(energies), "counts": np.array(counts)}


# ------------------------------------------------------------------------- what a pass cannot do without

def _energy_work(nq, nov, k):
    # R in once; the symmetric products (half of 2 NQ^2 nov) and the Cholesky factors of each point
    return 8.0 * nq * nov, k * (1.0 * nq * nq * nov + nq ** 3 / 3.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_energy_work(nq, no * nv, k) for nq, no, nv, k in _fragments(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    nq, nov = case["nq"], case["no"] * case["nv"]
    if kind == "mbe":
        b = f = 0.0
        for q, no, nv in _subsystems(case):
            pb, pf = _energy_work(q, no * nv, case["k"])
            g = min(3 * q, no * nv)  # guess vectors: the ring operator applied to them and to as many again
            b += pb
            f += pf + 2 * 4.0 * case["k"] * q * no * nv * g
        return {"bytes": b, "flops": f}
    if kind == "exchange":
        nt = case["nt"]
        pair = 1.0 * (case["no"] * (case["no"] + 1)) * nq * case["nv"] * nt * 2
        return {"bytes": 8.0 * nov * (nq + nt), "flops": 2 * pair + 2.0 * nov * nt * (nq + 2 * nt)}
    if kind == "pno":
        ng, nt = case["ng"], case["nt"]
        pairs = case["no"] * (case["no"] + 1) / 2
        return {"bytes": 8.0 * (ng * (nq + case["no"] + case["nv"]) + nov * nt),
                "flops": pairs * 2.0 * case["nv"] ** 2 * nt + 2.0 * ng * nq * nov}
    if kind == "thc":
        b, f = _energy_work(nq, nov, case["k"])
        return {"bytes": 8.0 * case["ng"] * (nq + case["no"] + case["nv"]), "flops": f + 2.0 * case["ng"] * nq * nov}
    b, f = _energy_work(nq, nov, case["k"])
    if kind == "pi":
        b += 8.0 * case["k"] * nq * nq
    elif kind in ("grad", "autograd"):
        b += 8.0 * nq * nov
        f += case["k"] * 2.0 * nq * nq * nov
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Four times what this path shows (rel: 2-norm, max: worst entry over the root mean square)."""
    kind = case["kind"]
    if kind == "pno":
        return {"rel": 1e-9}  # FP64; eigenvector bases of nearly equal PNO occupations may turn
    if case["prec"] == "split":
        # bf16 hi/lo operands with FP32 accumulation against FP64: up to 1.5e-6 over Pi, 6.4e-7 over dE/dR and
        # the energies, 1.1e-6 over the exchange energies; single entries of Pi and dE/dR 7.2e-5 of their rms
        return {"rel": 6e-6, "max": 3e-4}
    if kind == "mbe":
        return {"rel": 1e-10}  # one unit in the last place of R moves the exchange energies by 1e-11
    if kind == "exchange":
        return {"rel": 1e-9}  # the Lyapunov equation is solved to 1e-10
    # FP64 sums in another order: 3.3e-15 over E(u) and Pi, single entries of Pi 8e-15 of its rms; E_c, whose
    # high-frequency terms are differences of nearly equal log-determinants and traces, up to 4.9e-13
    return {"rel": 2e-12, "max": 1e-10}


# --------------------------------------------------------------------------------- 64-bit values

def _chi(d, u):
    return d / (d * d + u * u)


def _pi_exact(R, d, u):
    return 4.0 * (R * _chi(d, u)[None, :]) @ R.T


def _eu_exact(pi):
    L = torch.linalg.cholesky(pi + torch.eye(pi.shape[0], dtype=pi.dtype, device=pi.device))
    return float(2.0 * torch.log(torch.diagonal(L)).sum() - torch.trace(pi))


def _energy_exact(R, eo, ev, x, w):
    d = _gaps(eo, ev)
    eu = np.array([_eu_exact(_pi_exact(R, d, float(u))) for u in x])
    return math.fsum((w * eu).tolist()) / (2.0 * math.pi), eu


def _grad_exact(R, eo, ev, x, w):
    no, nv = len(eo), len(ev)
    d = _gaps(eo, ev)
    dR, dD, ec = torch.zeros_like(R.T).T, torch.zeros_like(d), 0.0
    for u, wu in zip(x, w):
        u, f = float(u), float(wu) / (2.0 * math.pi)
        pi = _pi_exact(R, d, u)
        ec += f * _eu_exact(pi)
        eye = torch.eye(pi.shape[0], dtype=pi.dtype, device=pi.device)
        MR = -torch.cholesky_solve(pi, torch.linalg.cholesky(pi + eye)) @ R  # ((1 + Pi)^-1 - 1) R
        dR += (8.0 * f) * _chi(d, u)[None, :] * MR
        dD += (4.0 * f) * (R * MR).sum(0) * (u * u - d * d) / (d * d + u * u) ** 2
    by_orbital = dD.reshape(no, nv)
    return ec, dR, -by_orbital.sum(1), by_orbital.sum(0)


def _exchange_exact(R, U, A, eo, ev):
    no, nv, nt = len(eo), len(ev), len(A)
    d = _gaps(eo, ev)
    At = torch.from_numpy(A).cuda()
    RU = R @ U
    Ukl, Dkl = RU.T @ RU, U.T @ (d[:, None] * U)
    right = At[:, None] * Dkl + Dkl * At[None, :]
    B = Dkl + 2.0 * Ukl + 4.0 * Ukl * At[None, :]
    # B^T X + X B = right: the symmetric part of B solved in its eigenbasis, the rest by residual correction
    mu, Q = torch.linalg.eigh(0.5 * (B + B.T))
    X = torch.zeros((nt, nt), dtype=R.dtype, device=R.device)
    for _ in range(30):
        res = right - B.T @ X - X @ B
        X = X + Q @ ((Q.T @ res @ Q) / (mu[:, None] + mu[None, :])) @ Q.T
    sosex = mbpt3 = 0.0
    UX = U @ X
    block = lambda M, i: M[nv * i:nv * (i + 1)]  # noqa: E731
    for i in range(no):
        for j in range(i + 1):
            f = 1.0 if i == j else 2.0
            Wij = R[:, nv * i:nv * (i + 1)] @ block(U, j)
            Rj = R[:, nv * j:nv * (j + 1)]
            sosex -= f * (Wij * (Rj @ block(U, i)) * At[None, :]).sum()
            mbpt3 -= f * (Wij * (Rj @ block(UX, i))).sum()
    return {"sosex": float(sosex), "mbpt3": float(mbpt3)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pno":
        return None  # pair by pair PNO truncation: minutes of small decompositions in plain torch
    s = prepare(case, seed)
    if kind == "energy":
        ec, eu = _energy_exact(*s["sys"])
        return {"ec": ec, "eu": eu}
    if kind == "pi":
        R, eo, ev, x, w = s["sys"]
        ec, eu = _energy_exact(R, eo, ev, x, w)
        d = _gaps(eo, ev)
        return {"pi": torch.stack([_pi_exact(R, d, float(u)) for u in x]), "ec": ec, "eu": eu}
    if kind == "batch":
        parts = [_energy_exact(*t) for t in s["systems"]]
        return {"ec": np.array([p[0] for p in parts]), "eu": [p[1] for p in parts]}
    if kind in ("grad", "autograd"):
        R, eo, ev, x, w = s["sys"]
        ec, dR, dO, dV = _grad_exact(R.detach(), eo, ev, x, w)
        if kind == "grad":
            return {"ec": ec, "dR": dR, "dO": dO, "dV": dV}
        return {"ec": ec, "grads": [dR, dO, dV]}
    if kind == "mbe":
        # the RPA energies on the driver's own grid; the amplitudes' random subspace has no 64-bit value
        sets = [(np.concatenate([eo, ev]), len(eo), len(ev)) for _, eo, ev in s["subsystems"]]
        x, w = _package().freq_grid_mbe(sets, nfixed=case["k"])
        ec = np.array([_energy_exact(R, eo, ev, x, w)[0] for R, eo, ev in s["subsystems"]])
        return {"freqs": None, "weights": None, "ec": ec, "ex": None, "eig_rpa": None, "nt": None,
                "common_thresh": None}
    if kind == "exchange":
        return _exchange_exact(s["R"], s["U"], s["A"], s["eo"], s["ev"])
    Z, Xa, Xi = s["factors"]
    kr = (Xi[:, :, None] * Xa[:, None, :]).reshape(case["ng"], -1)  # ai = a + NVirt * i
    ec, eu = _energy_exact(Z.T @ kr, s["eo"], s["ev"], *s["grid"])
    return {"ec": ec, "eu": eu}
