"""Sector enumeration where its filter, its warp queues and its chunks of 64
candidates can go wrong: one candidate up to many warps, ragged ends, 32- and
64-bit states, groups with and without rotations to filter by, momenta whose
characters reject symmetric states.  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nup,kw", [
    (6, 6, dict(kblock=0)), (6, None, dict(kblock=0)),                      # 1 and 64 candidates
    (17, None, dict(kblock=0)), (13, None, dict(kblock=4)),                 # every filling
    (20, 10, dict(kblock=0, pblock=1, zblock=1)), (20, 10, dict(kblock=10, pblock=-1, zblock=-1)),
    (19, 7, dict(kblock=3)), (18, 9, dict(pblock=1, zblock=-1)),            # 50,388; no rotations
    (32, 5, dict(kblock=16, pblock=1)), (18, 9, dict(kblock=3, a=2, zblock=1)),
    (2, 1, dict(kblock=0)), (3, 2, dict(kblock=1)), (9, 1, dict(kblock=2)), (9, 8, dict(kblock=2)),   # few odd ones
    (24, 9, dict(kblock=12, pblock=1)), (33, 4, dict(kblock=0, pblock=-1)), (40, 3, dict(kblock=20)), (36, 4, dict(pblock=1))])   # 64-bit states
def test_matches_oracle(qs, ora, L, nup, kw):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **kw)
    ref = ora.RepBasis(L, nup=nup, pauli=False, **kw)
    assert np.array_equal(b.orbit_minima(), ref.states)
    assert np.array_equal(b.index_array(b.states), np.arange(b.Ns))


@pytest.mark.parametrize("L,nup,q", [(18, 9, 0), (18, None, 3), (34, 3, 2)])
def test_general_maps(qs, L, nup, q):
    """The translation as a general site map gives the chain's sector."""
    shift = [(i + 1) % L for i in range(L)]
    g = qs.SpinBasisGeneral(L, nup=nup, pauli=False, T=(shift, q))
    c = qs.SpinBasis1D(L, nup=nup, pauli=False, kblock=q)
    assert np.array_equal(np.sort(g.states), np.sort(c.states)) and g.Ns == c.Ns
