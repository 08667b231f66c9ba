"""The particle-hole corrections with the pairs of an orbital in batches, against the same pairs one by one
(a workspace cap that leaves no room for batches)."""
import numpy as np
import pytest

from oracle import rpa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, cutoff", [
    ((120, 30, 5, 16, 24), 1e-10),      # every orbital kept: one by one, 2 n columns exceed the scratch
    ((201, 45, 6, 21, 50), 1e-3),       # few orbitals kept, odd sizes
    ((300, 60, 16, 256, 300), 1e-10),   # 70 MB per pair: 15 of the first orbital's 16 pairs fit in a batch
])
def test_batches_equal_single_pairs(pkg, shape, cutoff):
    # both forms sum the same products in another order: sums of at most 1e5 terms of either sign, each
    # rounded at 2^-53, and terms down to a thousandth of their parts
    ng, nq, no, nv, nt = shape
    Z, Xa, Xi, _, _ = O.make_thc_factors(ng, nq, no, nv, 44)
    rng = np.random.default_rng(144)
    U, _ = np.linalg.qr(rng.standard_normal((no * nv, nt)))
    A = -0.2 * rng.uniform(size=nt)
    with pkg.Handle(0) as h:
        free, stats = h.jctc2024(Z, Xi, Xa, U, A, cutoff_pno=cutoff)
        used = h.workspace_bytes()[0]
    with pkg.Handle(0) as h:
        h.set_workspace_limit(used - 1)
        capped, stats1 = h.jctc2024(Z, Xi, Xa, U, A, cutoff_pno=cutoff)
        assert h.workspace_bytes()[0] < used
    np.testing.assert_array_equal(stats, stats1)
    np.testing.assert_allclose(capped, free, rtol=1e-10, atol=1e-14)
