"""The engine's tiles (rows per BLAS block, slices per product block) follow the
slot's rows: ground states of sectors on both sides of each rule's edge."""
import numpy as np
import pytest

from models import j1j2, to_terms

pytestmark = pytest.mark.gpu

# (sites, sector) -> rows: one block of fewer than 768 rows, a partial second
# block, 304 blocks of more than 768 rows, and more than 20,000 slices (two
# slices per warp in the product)
SECTORS = [(16, dict(kblock=0, pblock=1, zblock=1)),
           (18, dict(kblock=0, pblock=1)),
           (27, dict(kblock=0, pblock=1)),
           (28, dict(kblock=0, pblock=1))]


@pytest.mark.parametrize("precision", ["fp64", "fp64df"])
@pytest.mark.parametrize("L,sym", SECTORS)
def test_ground_state_residual(qs, L, sym, precision, monkeypatch):
    # the graph-replayed step for every size (small slots would take the cluster step)
    monkeypatch.setenv("QS_CLUSTER_STEP", "0")
    b = qs.SpinBasis1D(L, nup=L // 2, pauli=False, **sym)
    terms = to_terms(qs, j1j2(L, J2=0.4))
    H = qs.Hamiltonian(b, terms)
    vals, vecs = qs.eigsh(H, k=1, tol=1e-12, precision=precision)
    v = vecs[:, 0]
    # the residual by the matrix-free FP64 product: the Ritz bound is 1e-12 |E|,
    # the vector's own rounding (48 bits in double-float) times ||H|| < 2 L below 2e-12
    r = qs.QuantumLinearOperator(b, terms).dot(v) - vals[0] * v
    assert abs(np.linalg.norm(v) - 1) < 1e-12
    assert np.linalg.norm(r) < 1e-10
