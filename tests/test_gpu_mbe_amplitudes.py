"""The amplitudes of the many-body driver on the device: no query of the free memory for small ones, and
the host's memory when the solver finds no room beside them."""
import numpy as np
import pytest

from oracle import rpa_oracle as O

pytestmark = pytest.mark.gpu


def _dimer():
    import torch
    out = []
    for nq, no, nv, seed in ((60, 4, 20, 1), (30, 2, 10, 2), (30, 2, 10, 3)):
        s = O.make_system(nq, no, nv, seed, decay=20.0, lam0=0.8)
        R = torch.from_numpy(np.ascontiguousarray(s.R.T)).cuda().T
        out.append((R, s.eps_o, s.eps_v))
    return out


def test_small_amplitudes_ask_for_no_memory_figures(handle, monkeypatch):
    import torch
    subs = _dimer()
    ref = handle.mbe_beyond_rpa(subs, 2, nfixed=8)

    def refuse(*a, **k):
        raise AssertionError("free memory queried")

    monkeypatch.setattr(torch.cuda, "mem_get_info", refuse)
    got = handle.mbe_beyond_rpa(subs, 2, nfixed=8)
    assert got["nt"] == ref["nt"] and np.array_equal(got["ex"], ref["ex"])


def test_solver_without_room_beside_the_amplitudes(handle, pkg, monkeypatch):
    subs = _dimer()
    ref = handle.mbe_beyond_rpa(subs, 2, nfixed=8)
    solve, refused = handle.dring_t2, []

    def short_of_memory(*a, u_out=None, **k):
        if u_out is not None:
            refused.append(1)
            raise pkg.RPAError(pkg.RPA_ERR_OOM, "no room")
        return solve(*a, **k)

    monkeypatch.setattr(handle, "dring_t2", short_of_memory)
    got = handle.mbe_beyond_rpa(subs, 2, nfixed=8)
    assert len(refused) == 3
    assert got["nt"] == ref["nt"] and np.array_equal(got["ex"], ref["ex"])
    monkeypatch.setattr(handle, "dring_t2", lambda *a, **k: (_ for _ in ()).throw(pkg.RPAError(pkg.RPA_ERR_NOT_SPD)))
    with pytest.raises(pkg.RPAError):
        handle.mbe_beyond_rpa(subs, 2, nfixed=8)
