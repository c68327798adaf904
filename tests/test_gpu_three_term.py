"""The three-term step (real recurrence coefficients) on both step forms, real
and complex matrices, every storage: evolved states against the dense exponential."""
import numpy as np
import pytest
import scipy.linalg as sla

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["0", "1"])
@pytest.mark.parametrize("precision,bound", [("fp64", 2e-11), ("fp64df", 2e-11), ("fp32", 2e-4)])
@pytest.mark.parametrize("L,sym,imag", [(12, dict(kblock=0, pblock=1), False), (11, dict(kblock=3), False),
                                        (6, dict(), True)])
def test_against_dense(qs, ora, monkeypatch, L, sym, imag, precision, bound, cluster):
    """bound: the step tolerance 1e-12 over the run's steps and rounding of the
    storage (2^-46 of the double-float sums, 2^-23 in single) times the products."""
    monkeypatch.setenv("QS_CLUSTER_STEP", cluster)
    b = qs.SpinBasis1D(L, pauli=True, **sym)
    H = qs.Hamiltonian(b, models.to_terms(qs, models.tfim(L)))
    D = ora.RefBasis(L, pauli=True, **sym).dense(ora.consolidate_terms(models.tfim(L)))
    v = models.seeded(b.Ns, complex_=True)
    v /= np.linalg.norm(v)
    times = [0.25, 1.0]
    tol = 1e-12 if precision != "fp32" else 1e-6
    got = qs.evolve(H, v, 0.0, times, imag_time=imag, tol=tol, krylov_dim=14, precision=precision)
    for i, t in enumerate(times):
        want = sla.expm((-t if imag else -1j * t) * D) @ v
        if imag:   # imaginary time normalises
            want /= np.linalg.norm(want)
        assert np.linalg.norm(got[:, i] - want) <= bound * np.linalg.norm(want), (i, t)
