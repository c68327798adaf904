"""A coupling that is not a number reaches the rows that it acts on, and no other."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["QuantumLinearOperator", "Hamiltonian"])
@pytest.mark.parametrize("at", [0, 4])
def test_nan_coupling(qs, form, at):
    L, nup = 8, 4
    b = qs.SpinBasis1D(L, nup=nup, pauli=False)
    bonds = [(0.5 + 0.1 * (i % 2), i, i + 1) for i in range(1, L)]
    good = [c for k, c in enumerate(bonds) if k != at]
    bad = [(float("nan"),) + c[1:] if k == at else c for k, c in enumerate(bonds)]
    make = getattr(qs, form)
    x = models.seeded(b.Ns)
    want = make(b, models.to_terms(qs, [("+-", good), ("-+", good)])).dot(x)
    got = make(b, models.to_terms(qs, [("+-", bad), ("-+", bad)])).dot(x)
    # site i is bit i - 1: the bond acts on the states whose two bits differ
    s = np.asarray(b.states, dtype=np.uint64)
    hit = ((s >> np.uint64(at)) ^ (s >> np.uint64(at + 1))) & np.uint64(1) == 1
    assert np.array_equal(np.isnan(got), hit)
    assert np.allclose(got[~hit], want[~hit], rtol=0, atol=1e-15 * 8)
