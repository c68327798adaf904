"""Extremal pairs on both step forms, real and complex, with and without a large
constant on the diagonal: the Ritz values against the dense spectrum and the
vectors' residuals."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["0", "1"])
@pytest.mark.parametrize("precision", ["fp64", "fp64df"])
@pytest.mark.parametrize("L,sym,shift", [(12, dict(kblock=0, pblock=1), 0.0), (13, dict(kblock=2), 0.0),
                                         (12, dict(kblock=0, pblock=1), 1e3), (13, dict(kblock=2), -1e3)])
def test_extremal_pairs(qs, ora, monkeypatch, L, sym, shift, precision, cluster):
    """shift: a constant on the diagonal far above ||H||, where the unshifted
    step would cancel almost everything in its first pass."""
    monkeypatch.setenv("QS_CLUSTER_STEP", cluster)
    nup = L // 2
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    spec = models.j1j2(L, 1.0, 0.37) + ([("I", [(shift / L, i) for i in range(1, L + 1)])] if shift else [])
    H = qs.Hamiltonian(b, models.to_terms(qs, spec))
    D = ora.RefBasis(L, nup=nup, pauli=False, **sym).dense(ora.consolidate_terms(models.j1j2(L, 1.0, 0.37)))
    w = np.linalg.eigvalsh(D) + shift
    vals, vecs = qs.eigsh(H, k=3, tol=1e-13, precision=precision)
    size = np.abs(w).max()
    # Ritz bound 1e-13 |theta|, products of 48 bits (double-float) on ||H||
    assert np.max(np.abs(vals - w[:3])) <= 1e-12 * size
    r = (D @ vecs + shift * vecs) - vecs * vals
    assert np.max(np.linalg.norm(r, axis=0)) <= 1e-11 * size
    assert np.max(np.abs(vecs.conj().T @ vecs - np.eye(3))) <= 1e-12
