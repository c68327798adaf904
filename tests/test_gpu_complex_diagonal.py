"""A complex diagonal set on a real matrix-free operator acts on complex vectors."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nup,sym", [(8, 4, {}), (10, 5, dict(kblock=0, pblock=1)), (9, None, {}), (34, 2, dict(kblock=0))])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_complex_diagonal(qs, L, nup, sym, precision):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    op = qs.QuantumLinearOperator(b, models.to_terms(qs, models.xxz(L)))
    x = models.seeded(b.Ns, complex_=True)
    y = np.zeros(b.Ns, dtype=np.complex128)
    base = op.mul(y, x, precision=precision).copy()
    d = models.seeded(b.Ns, seed=7, complex_=True)
    op.set_diagonal(d)
    # one product and one addition on values of a few units
    tol = 1e-14 if precision == "fp64" else 1e-5
    scale = np.abs(x).max() * (np.abs(d).max() + L)
    assert np.max(np.abs(op.mul(y, x, precision=precision) - (base + d * x))) <= tol * scale
    assert np.max(np.abs(op.conj().mul(y, x, precision=precision) - (base + d.conj() * x))) <= tol * scale
    # and a real one again
    op.set_diagonal(d.real)
    assert np.max(np.abs(op.mul(y, x, precision=precision) - (base + d.real * x))) <= tol * scale
