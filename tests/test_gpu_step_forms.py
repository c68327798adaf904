"""Both sides of each limit between the cluster step and the graph replay: the
eigenvalues of the form that the size picks are those of the other one."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nup,sym,precision,rows", [
    (17, 8, {}, "fp64", 24310), (17, 7, {}, "fp64", 19448), (17, 8, {}, "fp64df", 24310),
    (20, 9, dict(kblock=3), "fp64", 8398),
    (21, 9, dict(kblock=3), "fp64df", 14000), (21, 10, dict(kblock=3), "fp64df", 16796)])
def test_forms_agree(qs, monkeypatch, L, nup, sym, precision, rows):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    assert b.Ns == rows
    H = qs.Hamiltonian(b, models.to_terms(qs, models.xxz(L, 1.0, 0.8)))
    got = {}
    for form in ("", "0", "1"):
        monkeypatch.setenv("QS_CLUSTER_STEP", form)
        got[form] = qs.eigsh(H, k=2, tol=1e-12, precision=precision, return_eigenvectors=False)
    # each solve is within its Ritz bound, 1e-12 |theta|, of the spectrum
    for form in ("0", "1"):
        assert np.max(np.abs(got[form] - got[""])) <= 4e-12 * np.abs(got[""]).max(), form
