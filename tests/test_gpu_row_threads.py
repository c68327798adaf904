"""Products and assemblies of two sectors from two threads: the sectors share a
kernel and need different amounts of its shared memory."""
import ctypes
import threading

import numpy as np
import pytest

import models

pytestmark = pytest.mark.gpu

def together(work):
    errors, gate = [], threading.Barrier(len(work))

    def run(w):
        try:
            gate.wait(30)
            w()
        except Exception as e:   # noqa: BLE001 (reported below)
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=(w,)) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:2]


def test_products(qs):
    """Many columns in a call, so that the launches of both threads follow one
    another closely: tables of 16.4 and 19.5 KB."""
    torch = pytest.importorskip("torch")
    from qsgpu import _lib
    lib = _lib.load()
    one, zero = np.array([1.0, 0.0]), np.zeros(2)
    work, checks = [], []
    for L, nup, cols in [(32, 4, 1500), (32, 5, 400)]:
        b = qs.SpinBasis1D(L, nup=nup, pauli=False)
        op = qs.QuantumLinearOperator(b, models.to_terms(qs, models.xxz(L)))
        x = torch.zeros((cols, b.Ns), dtype=torch.float64, device="cuda")
        x[:] = torch.from_numpy(models.seeded(b.Ns)).cuda()
        y = torch.zeros_like(x)
        torch.cuda.synchronize()

        def loop(op=op, x=x, y=y, cols=cols):
            for _ in range(6):
                _lib.check(lib.qs_op_matvec(op._h, 0, _lib.ptr(one), ctypes.c_void_p(x.data_ptr()), 0, _lib.ptr(zero),
                                            ctypes.c_void_p(y.data_ptr()), 0, cols, _lib.QS_MEM_DEVICE))

        work.append(loop)
        checks.append((op, x, y))
    together(work)
    torch.cuda.synchronize()
    for op, x, y in checks:
        want = torch.from_numpy(op.dot(x[0].cpu().numpy())).cuda()
        assert torch.equal(y, want.expand_as(y))


def test_assemblies(qs):
    bases = [qs.SpinBasis1D(L, nup=nup, pauli=False) for L, nup in ((32, 5), (32, 6))]
    terms = models.to_terms(qs, models.xxz(32))
    want = [qs.Hamiltonian(b, terms).nnz for b in bases]
    nnz = [[], []]

    def loop(i):
        for _ in range(60):
            nnz[i].append(qs.Hamiltonian(bases[i], terms).nnz)

    together([lambda: loop(0), lambda: loop(1)])
    assert [set(v) for v in nnz] == [{w} for w in want]
