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
