"""Assembled operators whose terms leave the particle sector (check_pcon off):
the images of another particle number have no column, in the product and in the
exported matrix, whichever lookup finds the columns."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


# the split ranks (no symmetry, 32-bit states), the direct table, complex
# characters, 64-bit states, and few or almost only particles
@pytest.mark.parametrize("L,nup,sym", [(12, 5, {}), (12, 5, dict(kblock=0, pblock=1)), (12, 6, dict(kblock=0, zblock=1)),
                                       (13, 6, dict(kblock=3)), (34, 2, {}), (34, 3, dict(kblock=0)), (32, 1, {}),
                                       (20, 19, {}), (20, 19, dict(kblock=0)), (16, 16, {})])
def test_assembled_outside_the_sector(qs, L, nup, sym):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    spec = models.j1j2(L, 1.0, 0.45)
    # raises or lowers one particle, and a hop that creates one more
    field = [("x", [(0.3, i) for i in range(1, L + 1)])] + (
        [] if "zblock" in sym else [("++-", [(0.2, i, i % L + 1, (i + 1) % L + 1) for i in range(1, L + 1)]),
                                    ("--+", [(0.2, i, i % L + 1, (i + 1) % L + 1) for i in range(1, L + 1)])])
    if "pblock" in sym:
        field = field[:1]
    kept = qs.Hamiltonian(b, models.to_terms(qs, spec))
    H = qs.Hamiltonian(b, models.to_terms(qs, spec + field), check_pcon=False, check_herm=False)
    assert H.assembled and kept.assembled
    x = models.seeded(b.Ns, complex_=H.dtype == np.complex128)
    assert H.nnz == kept.nnz
    assert np.array_equal(H.dot(x), kept.dot(x))
    A, B = H.tocsr(), kept.tocsr()
    assert abs(A - B).nnz == 0
