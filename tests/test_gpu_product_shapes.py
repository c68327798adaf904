"""The assembled product's shape follows from the rows and their mean length:
sectors on both sides of the rule's lines, without an override, against both
shapes."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


# complex FP64 at 100,000 rows; short rows at a million; fixed point at 200,000
@pytest.mark.parametrize("model,L,nup,sym,precision,rows", [
    ("j1j2", 24, 11, dict(kblock=5), "fp64", 104006), ("j1j2", 23, 11, dict(kblock=5), "fp64", 58786),
    ("xxz", 26, 9, dict(kblock=0), "fp64", 120175), ("xxz", 24, 10, {}, "fp64", 1961256),
    ("j1j2", 28, 12, dict(kblock=0, pblock=1), "fp64fx", None), ("j1j2", 26, 13, dict(kblock=0, pblock=1, zblock=1), "fp64fx", 101340)])
def test_rule_and_both_shapes(qs, monkeypatch, model, L, nup, sym, precision, rows):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    assert rows is None or b.Ns == rows
    spec = models.j1j2(L, 1.0, 0.45) if model == "j1j2" else models.xxz(L)
    H = qs.Hamiltonian(b, models.to_terms(qs, spec))
    x = models.seeded(b.Ns, complex_=H.dtype == np.complex128)
    got = []
    for v in ("", "0", "1"):
        monkeypatch.setenv("QS_SELL_VARIANT", v)
        got.append(H.dot(x, precision=precision))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
