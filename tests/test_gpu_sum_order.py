"""The order in which a solve's sums are added.  An eigenvector's sign follows
the last bits of the projected matrix, so the order is part of the output: the
norm of a start vector against the order restated in numpy, bit for bit, and
signs of ground states that another order turns over."""
import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu

BLOCK, LANES = 4096, 256


def butterfly(v):
    """Totals of 32 lanes, added at xor distances 16, 8, 4, 2, 1 (axis -1)."""
    for o in (16, 8, 4, 2, 1):
        v = v + v[..., np.arange(32) ^ o]
    return v[..., 0]


def sum_of_squares(x):
    """Blocks of 4,096 rows: lane l adds rows l, l + 256, ..., then the lanes of
    each of eight warps, the warps, and the blocks (256 lanes again)."""
    nb = -(-x.size // BLOCK)
    sq = np.zeros(nb * BLOCK)
    sq[:x.size] = x * x          # exact: x has 24-bit mantissas, so a fused
    sq = sq.reshape(nb, BLOCK // LANES, LANES)   # multiply-add rounds the same
    acc = np.zeros((nb, LANES))
    for k in range(BLOCK // LANES):
        acc = acc + sq[:, k]
    warps = butterfly(acc.reshape(nb, 8, 32))
    block = np.zeros(nb)
    for q in range(8):
        block = block + warps[:, q]
    lanes = np.zeros(LANES)
    for b0 in range(0, nb, LANES):
        part = block[b0:b0 + LANES]
        lanes[:part.size] = lanes[:part.size] + part
    w = butterfly(lanes.reshape(8, 32))
    t = 0.0
    for q in range(8):
        t = t + w[q]
    return t


@pytest.mark.parametrize("L,nup", [(8, 3), (12, 6), (16, 7), (18, 8), (20, 10), (24, 9)])   # 56 .. 1,307,504 rows
def test_norm_of_a_start_vector(qs, L, nup):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False)
    H = qs.Hamiltonian(b, models.to_terms(qs, models.xxz(L)))
    x = np.random.default_rng(L).standard_normal(b.Ns).astype(np.float32).astype(np.float64)
    from qsgpu.tools import _LanczosSet
    q0 = _LanczosSet(H, x, 2, full_ortho=True).rows(0)[0]
    assert np.array_equal(q0, x * (1.0 / np.sqrt(sum_of_squares(x))))


def sign_of(qs, model, L, nup, sym, form, coupling, seed, precision="fp64", which="SA"):
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    spec = models.j1j2(L, 1.0, coupling) if model == "j1j2" else models.xxz(L, 1.0, coupling)
    H = (qs.Hamiltonian if form == "H" else qs.QuantumLinearOperator)(b, models.to_terms(qs, spec))
    rng = np.random.default_rng(seed)
    v0 = rng.standard_normal(b.Ns)
    if H.dtype == np.complex128:
        v0 = v0 + 1j * rng.standard_normal(b.Ns)
    vec = qs.eigsh(H, k=1, tol=1e-12, v0=v0, precision=precision, which=which)[1][:, 0]
    return np.sign((np.random.default_rng(5).standard_normal(b.Ns) @ vec).real)


EVEN = dict(kblock=0, pblock=1, zblock=1)


# Start vectors, of a hundred, whose eigenvector turns over when the blocks of
# the sums have other sizes, with the sign of 4,096-row blocks; the coupling is
# 0.2 + 0.25 (i + 0.5) / n.
@pytest.mark.parametrize("L,sym,i,n,seed,precision,sign", [
    (20, EVEN, 3, 4, 3002, "fp64", -1), (26, EVEN, 2, 3, 2003, "fp64", -1),
    (28, EVEN, 1, 3, 1003, "fp64", 1), (28, EVEN, 1, 3, 1004, "fp64", -1), (28, EVEN, 1, 3, 1008, "fp64", 1),
    (16, dict(kblock=3), 1, 3, 1011, "fp64", -1),
    (26, EVEN, 1, 2, 1008, "fp64df", -1), (22, EVEN, 0, 2, 7, "fp32", 1), (26, EVEN, 1, 2, 1001, "fp32", -1)])
def test_signs_of_ground_states(qs, L, sym, i, n, seed, precision, sign):
    c = 0.2 + 0.25 * (i + 0.5) / n
    assert sign_of(qs, "j1j2", L, L // 2, sym, "H", c, seed, precision) == sign


# ... and when slots of 8,193 to 32,768 rows change between the cluster step and
# the graph replay
@pytest.mark.parametrize("model,L,nup,sym,i,n,seed,precision,which,sign", [
    ("j1j2", 20, 10, dict(kblock=3), 1, 3, 1009, "fp64", "SA", -1),
    ("j1j2", 20, 10, dict(kblock=3), 2, 3, 2008, "fp64", "SA", 1),
    ("j1j2", 21, 10, dict(kblock=2), 0, 3, 3, "fp64", "SA", -1),
    ("j1j2", 21, 10, dict(kblock=2), 2, 3, 2010, "fp64", "SA", 1),
    ("xxz", 17, 8, {}, 1, 3, 1010, "fp64", "SA", -1), ("xxz", 17, 8, {}, 1, 3, 1014, "fp64", "SA", 1),
    ("j1j2", 24, 12, EVEN, 0, 2, 7, "fp64df", "SA", -1), ("j1j2", 24, 12, EVEN, 1, 2, 1008, "fp64", "LA", 1)])
def test_signs_between_the_step_forms(qs, model, L, nup, sym, i, n, seed, precision, which, sign):
    c = 0.2 + 0.25 * (i + 0.5) / n
    assert sign_of(qs, model, L, nup, sym, "H", c, seed, precision, which) == sign


# one CTA's slices empty, eight and sixteen CTAs, both ends of their ranges
@pytest.mark.parametrize("precision", ["fp64", "fp64df", "fp32"])
@pytest.mark.parametrize("L,nup,sym,rows", [
    (8, 4, {}, 70), (14, 7, EVEN, 85), (14, 6, dict(kblock=3), 212), (22, 11, EVEN, 8359), (17, 8, {}, 24310),
    (20, 10, dict(kblock=3), 9225), (21, 10, dict(kblock=2), 16796), (33, 3, {}, 5456), (22, 11, dict(kblock=1), 32065)])
def test_step_forms_give_the_same_bits(qs, monkeypatch, L, nup, sym, rows, precision):
    """Solves of up to 32,768 rows: the cluster step, the graph replay and the rule."""
    b = qs.SpinBasis1D(L, nup=nup, pauli=False, **sym)
    assert b.Ns == rows
    H = qs.Hamiltonian(b, models.to_terms(qs, models.j1j2(L, 1.0, 0.3)))
    got = []
    for form in ("", "0", "1"):
        monkeypatch.setenv("QS_CLUSTER_STEP", form)
        got.append(qs.eigsh(H, k=2, tol=1e-11, precision=precision))
    for vals, vecs in got[1:]:
        assert np.array_equal(vals, got[0][0]) and np.array_equal(vecs, got[0][1])


# ... and when the terms of the matrix-free product (operators of fewer than
# 4,096 rows) are rounded in another order
@pytest.mark.parametrize("L,sym,i,seed,sign", [
    (14, EVEN, 0, 4, 1), (14, EVEN, 1, 1014, 1), (14, EVEN, 2, 2013, 1), (14, EVEN, 3, 3008, -1),
    (18, EVEN, 0, 3, 1), (18, EVEN, 1, 1001, -1), (18, EVEN, 3, 3009, 1),
    (20, EVEN, 2, 2003, 1), (20, EVEN, 3, 3008, -1),
    (14, dict(kblock=2), 0, 18, -1), (14, dict(kblock=2), 1, 1003, -1), (14, dict(kblock=2), 2, 2015, 1),
    (14, dict(kblock=2), 3, 3007, -1), (14, dict(kblock=2), 3, 3017, -1)])
def test_signs_of_matrix_free_solves(qs, L, sym, i, seed, sign):
    assert sign_of(qs, "j1j2", L, L // 2, sym, "Q", 0.2 + 0.25 * (i + 0.5) / 4, seed) == sign
