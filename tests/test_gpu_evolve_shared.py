"""Evolution to several times shares the states that the times have in common:
each time's state equals the one it has alone, bit for bit."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


# a grid whose steps coincide, times that repeat, scattered ones, imaginary time;
# sizes on the cluster step and on the graph replay
@pytest.mark.parametrize("L,sym", [(12, dict(kblock=0, pblock=1)), (19, dict(kblock=0)), (22, dict(kblock=0, pblock=1))])
@pytest.mark.parametrize("times", [np.linspace(0.2, 2.0, 10), [0.5, 2.0, 0.5, 1.0], [0.3, 1.7, 0.91, 1.3, 0.02]])
@pytest.mark.parametrize("imag", [False, True])
def test_each_time_as_alone(qs, L, sym, times, imag):
    b = qs.SpinBasis1D(L, pauli=True, **sym)
    H = qs.Hamiltonian(b, models.to_terms(qs, models.tfim(L)))
    v = models.seeded(b.Ns, complex_=True)
    v /= np.linalg.norm(v)
    kw = dict(imag_time=imag, tol=1e-10, krylov_dim=12)
    together = qs.evolve(H, v, 0.0, times, **kw)
    for i, t in enumerate(times):
        assert np.array_equal(together[:, i], qs.evolve(H, v, 0.0, [t], **kw)[:, 0]), (i, t)


def test_columns_and_times_as_alone(qs):
    """Several start vectors at several times (one engine, one group per vector)."""
    L = 16
    b = qs.SpinBasis1D(L, pauli=True, kblock=0)
    H = qs.Hamiltonian(b, models.to_terms(qs, models.tfim(L)))
    V = np.stack([models.seeded(b.Ns, seed=s, complex_=True) for s in (1, 2, 3)], axis=1)
    times = np.linspace(0.25, 1.5, 6)
    kw = dict(tol=1e-10, krylov_dim=12)
    out = qs.evolve(H, V, 0.0, times, **kw)
    for c in range(3):
        for i, t in enumerate(times):
            assert np.array_equal(out[:, c, i], qs.evolve(H, V[:, c:c + 1], 0.0, [t], **kw)[:, 0, 0])
