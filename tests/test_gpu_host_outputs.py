"""Host outputs are prepared for the device's copy only where nothing is read
from them: adding to a page-locked output, products in place, and an output that
is not host memory."""
import ctypes

import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
def test_project_adds_to_its_output(qs, pinned):
    torch = pytest.importorskip("torch")
    from qsgpu import _lib
    b = qs.SpinBasis1D(21, nup=10, pauli=False, kblock=0, pblock=1)
    rows = qs.SpinBasis1D(21, nup=10, pauli=False).Ns
    v = models.seeded(b.Ns, complex_=True)
    base = models.seeded(rows, seed=3, complex_=True)
    want = np.zeros(rows, dtype=np.complex128)
    lib = _lib.load()
    _lib.check(lib.qs_basis_project_from(b._h, 1, _lib.ptr(v), _lib.ptr(want), 0, _lib.QS_MEM_HOST))
    out = torch.empty(rows, dtype=torch.complex128, pin_memory=pinned).numpy()
    for _ in range(5):
        out[:] = base
        _lib.check(lib.qs_basis_project_from(b._h, 1, _lib.ptr(v), _lib.ptr(out), 1, _lib.QS_MEM_HOST))
        assert np.max(np.abs(out - (base + want))) <= 4e-16 * 16   # one addition of values of a few units


@pytest.mark.parametrize("form", ["QuantumLinearOperator", "Hamiltonian"])
@pytest.mark.parametrize("pinned", [True, False])
def test_product_in_place(qs, form, pinned):
    torch = pytest.importorskip("torch")
    from qsgpu import _lib
    b = qs.SpinBasis1D(20, nup=10, pauli=False)
    op = getattr(qs, form)(b, models.to_terms(qs, models.xxz(20)))
    x = models.seeded(b.Ns)
    want = op.dot(x)
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    z = torch.empty(b.Ns, dtype=torch.float64, pin_memory=pinned).numpy()
    for _ in range(5):
        z[:] = x
        _lib.check(_lib.load().qs_op_matvec(op._h, 0, _lib.ptr(one), _lib.ptr(z), 0, _lib.ptr(zero), _lib.ptr(z), 0, 1,
                                            _lib.QS_MEM_HOST))
        assert np.array_equal(z, want)


def test_device_memory_as_a_host_output(qs):
    """An error, or the product where the copy takes it; not a crash."""
    torch = pytest.importorskip("torch")
    from qsgpu import _lib
    b = qs.SpinBasis1D(14, nup=7, pauli=False)
    op = qs.QuantumLinearOperator(b, models.to_terms(qs, models.xxz(14)))
    x = models.seeded(b.Ns)
    want = op.dot(x)
    y = torch.zeros(b.Ns, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    st = _lib.load().qs_op_matvec(op._h, 0, _lib.ptr(one), _lib.ptr(x), 0, _lib.ptr(zero), ctypes.c_void_p(y.data_ptr()), 0,
                                  1, _lib.QS_MEM_HOST)
    assert st != 0 or np.array_equal(y.cpu().numpy(), want)
    assert np.array_equal(op.dot(x), want)
