"""The diagonal's kernel at its edges: the chunk of 256 programs, strings that
touch a site twice, imaginary amplitudes, a user diagonal on top, single
precision and double-float copies; against the oracle."""
import itertools

import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


def spec_for(nprog, imag, twice):
    pairs = list(itertools.combinations(range(1, 25), 2))
    rng = np.random.default_rng(nprog)
    zz = [(float(c), i, j) for c, (i, j) in zip(rng.uniform(-1, 1, nprog), pairs[:nprog])]
    spec = [("zz", zz), ("+-", [(0.25, 1, 2)]), ("-+", [(0.25, 1, 2)])]
    if imag:
        spec.append(("z", [(0.5j, 3), (-0.125j, 24)]))
    if twice:
        spec.append(("zzz", [(0.75, 4, 4, 5)]))
    return spec


@pytest.mark.parametrize("nprog,imag,twice", [(1, False, False), (255, False, False), (256, False, False),
                                              (257, False, True), (276, True, False), (30, True, True)])
def test_matches_oracle(qs, ora, nprog, imag, twice):
    b = qs.SpinBasis1D(24, nup=2, pauli=False)
    spec = spec_for(nprog, imag, twice)
    user = models.seeded(b.Ns)
    H = qs.QuantumLinearOperator(b, models.to_terms(qs, spec), diagonal=user, check_herm=False)
    ref = ora.RefBasis(24, nup=2, pauli=False)
    D = ref.dense(ora.consolidate_terms(spec)) + np.diag(user)
    bound = nprog + 4
    x = models.seeded(b.Ns, complex_=True)
    # |diagonal| <= nprog / 4 + 2: rounding of at most nprog additions
    assert np.abs(H.dot(x) - D @ x).max() <= bound * 2.0 ** -50 * bound
    x32 = x.astype(np.complex64)
    assert np.abs(H.dot(x32) - D @ x32).max() <= bound * 2.0 ** -20
