"""The row walk of the matrix-free product and the assembly (live-program masks, orbit minimum by
windows, split rank tables) at the sizes where it can go wrong, against the
oracle's representative-space product."""
import os

import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


def all_pairs(L, seed=5):
    """Exchange between every pair of sites by distance: more than 128 programs from L = 12 on."""
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.2, 1.0, L)
    d = [d[min(k, L - k)] for k in range(L)]
    flips = [(0.5 * d[j - i], i, j) for i in range(1, L + 1) for j in range(i + 1, L + 1)]
    return [("+-", flips), ("-+", flips), ("zz", [(2 * c, i, j) for c, i, j in flips])]


# both ends of the window search (one window group, all four, an even split of
# 32 bits, three prime factors, a prime length), every kind of element code, the
# groups that keep the zero-run search (a = 2) and no translations at all
CASES = [
    (2, 1, dict(kblock=0), "j1j2"), (3, 1, dict(kblock=1), "j1j2"), (8, 4, dict(kblock=2, zblock=-1), "j1j2"),
    (9, 4, dict(kblock=4), "j1j2"), (16, 8, dict(kblock=8, pblock=-1, zblock=1), "j1j2"),
    (23, 3, dict(kblock=7), "j1j2"), (30, 4, dict(kblock=0, pblock=-1), "j1j2"), (30, 4, dict(kblock=10), "j1j2"),
    (31, 3, dict(kblock=30), "j1j2"), (32, 4, dict(kblock=0, pblock=1), "j1j2"), (32, 3, dict(kblock=31), "j1j2"),
    (33, 3, dict(kblock=2), "j1j2"), (12, None, dict(kblock=0, pblock=1, zblock=-1), "tfim"),
    (12, 6, dict(pblock=-1), "j1j2"), (12, 6, dict(zblock=1), "j1j2"), (12, 6, dict(pblock=1, zblock=-1), "j1j2"),
    (16, 8, dict(kblock=2, a=2), "j1j2"), (14, 7, dict(kblock=3), "pairs"), (14, 7, dict(kblock=0, pblock=1, zblock=1), "pairs"),
    (14, 7, dict(), "pairs"), (32, 3, dict(), "j1j2"), (33, 3, dict(), "j1j2"), (11, None, dict(kblock=4), "xyz"),
]


@pytest.mark.parametrize("L,nup,sym,model", CASES)
def test_row_walk_against_oracle(qs, ora, L, nup, sym, model):
    spec = {"j1j2": lambda: models.j1j2(L, 1.0, 0.45), "tfim": lambda: models.tfim(L), "pairs": lambda: all_pairs(L),
            "xyz": lambda: models.xyz_field(L)}[model]()
    pauli = model == "tfim"
    b = qs.SpinBasis1D(L, nup=nup, pauli=pauli, **sym)
    rep = ora.RepBasis(L, nup=nup, pauli=pauli, **sym)
    assert b.Ns == rep.Ns
    x = models.seeded(b.Ns, complex_=True)
    want = rep.matvec(ora.consolidate_terms(spec), x)
    scale = max(1.0, float(np.abs(want).max()))
    op = qs.QuantumLinearOperator(b, models.to_terms(qs, spec))
    # the summation order of the row, as the other products are held: 1e-13
    assert np.max(np.abs(op.dot(x) - want)) <= 1e-13 * scale
    if op.dtype == np.float64:
        assert np.max(np.abs(op.dot(x.real.copy()) - want.real)) <= 1e-13 * scale


@pytest.mark.parametrize("sym", [dict(kblock=0, pblock=1), dict(kblock=3), dict()])
def test_programs_outside_the_particle_sector(qs, sym):
    """With check_pcon off, states of another particle number have no column and
    drop out, whichever lookup would have found them."""
    L, nup = 12, 5
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    spec = models.j1j2(L, 1.0, 0.45)
    x = models.seeded(b.Ns, complex_=bool(sym.get("kblock")))
    field = [("x", [(0.3, i) for i in range(1, L + 1)])]
    kept = qs.QuantumLinearOperator(b, models.to_terms(qs, spec)).dot(x)
    op = qs.QuantumLinearOperator(b, models.to_terms(qs, spec + field), check_pcon=False)
    assert np.array_equal(op.dot(x), kept)
    old = os.environ.get("QS_RANK_MODE")
    os.environ["QS_RANK_MODE"] = "search"
    try:
        assert np.array_equal(op.dot(x), kept)
    finally:
        os.environ.pop("QS_RANK_MODE") if old is None else os.environ.update(QS_RANK_MODE=old)


def test_site_acted_on_twice(qs, ora):
    """Programs run by their characters (a site acted on twice) beside compiled ones."""
    L = 10
    b = qs.SpinBasis1D(L, pauli=False, kblock=0)
    ref = ora.RefBasis(L, pauli=False, kblock=0)
    sites = range(1, L + 1)
    spec = [("zx", [(0.7, i, i) for i in sites]), ("x", [(0.4, i) for i in sites])]
    x = models.seeded(b.Ns, complex_=True)
    got = qs.QuantumLinearOperator(b, models.to_terms(qs, spec), check_herm=False).dot(x)
    want = ref.qlo_matvec(ora.consolidate_terms(spec), x)
    assert np.max(np.abs(got - want)) <= 1e-13 * max(1.0, float(np.abs(want).max()))


# (the two-site chain's second-neighbour bond acts on one site twice: not assembled)
@pytest.mark.parametrize("L,nup,sym,model", CASES[1:])
def test_assembled_walk_against_matrix_free(qs, L, nup, sym, model):
    """The assembly walks the same transitions: its product (table values, the same
    order) agrees with the matrix-free one to rounding, and so does its export."""
    spec = {"j1j2": lambda: models.j1j2(L, 1.0, 0.45), "tfim": lambda: models.tfim(L), "pairs": lambda: all_pairs(L),
            "xyz": lambda: models.xyz_field(L)}[model]()
    b = qs.SpinBasis1D(L, nup=nup, pauli=model == "tfim", **sym)
    terms = models.to_terms(qs, spec)
    x = models.seeded(b.Ns, complex_=True)
    want = qs.QuantumLinearOperator(b, terms).dot(x)
    H = qs.Hamiltonian(b, terms)
    assert H.assembled
    scale = max(1.0, float(np.abs(want).max()))
    assert np.max(np.abs(H.dot(x) - want)) <= 1e-13 * scale
    assert np.max(np.abs(H.tocsr() @ x - want)) <= 1e-13 * scale


@pytest.mark.parametrize("L,nup,longest", [(24, 1, 5313), (11, None, 65536)])
def test_assembly_of_many_programs(qs, L, nup, longest):
    """More than 65,535 programs: assembled through CSR, kept in the sliced layout
    where the rows fit its lengths (nup = 1) and in CSR where they do not."""
    from itertools import combinations
    rng = np.random.default_rng(11)
    if nup:
        c = [(float(v), *ij, *kl) for ij in combinations(range(1, L + 1), 2)
             for kl in combinations([q for q in range(1, L + 1) if q not in ij], 2) for v in [rng.choice([0.25, 0.5])]]
        spec = [("+-zz", c), ("-+zz", c)]
    else:
        spec = []
        for nx in range(1, 9):
            for nz in range(0, 9 - nx):
                spec.append(("x" * nx + "z" * nz,
                             [(0.5, *xs, *zs) for xs in combinations(range(1, L + 1), nx)
                              for zs in combinations([q for q in range(1, L + 1) if q not in xs], nz)]))
    b = qs.SpinBasis1D(L, nup=nup, pauli=True)
    terms = models.to_terms(qs, spec)
    H = qs.Hamiltonian(b, terms)
    assert H.assembled and H.nnz >= longest * (b.Ns if nup is None else 1)
    x = models.seeded(b.Ns)
    want = qs.QuantumLinearOperator(b, terms).dot(x)
    # rows of up to 1.3e5 terms of the same size: n eps of the sum of magnitudes
    mag = H.nnz / b.Ns * 4 * np.abs(x).max()
    assert np.max(np.abs(H.dot(x) - want)) <= 1e-13 * mag
