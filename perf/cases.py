"""The work that users have qsgpu do, as cases that can be timed and checked.

Each case goes through the public entry points: the Python binding
(SpinBasis1D, QuantumLinearOperator, Hamiltonian, eigsh, evolve) or,
for vectors that live on the device, the C entry point qs_op_matvec that the
binding wraps.  Inputs come from the seed alone; exact() restates the
result in 64 bits with plain torch and numpy (its own enumeration of the
states, its own orbits and ranks, its own Lanczos and Chebyshev recursions).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "quspin.jl_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "quspin.jl_gb300"))

# products and kept basis vectors that a ground state at tol 1e-12 takes on these
# chains (nominal, for work() alone)
_SOLVE_PRODUCTS = 80
_SOLVE_BASIS = 20


# ------------------------------------------------------------------ the cases
def _case(kind, model, L, nup=-1, k=-1, p=0, z=0, form="linear_operator", dtype="float64", coupling=None, **more):
    """nup = -1: no particle number; k = -1: no momentum; p, z = 0: no parity, no spin flip.
    coupling: Delta of the XXZ chain, J2 of the J1-J2 chain, the field of the Ising chain."""
    if coupling is None:
        coupling = {"xxz": 0.5, "j1j2": 0.5, "tfim": 0.7}[model]
    return dict(kind=kind, model=model, L=L, nup=nup, k=k, p=p, z=z, form=form, dtype=dtype, coupling=coupling, **more)


def listed():
    return [
        # the smallest call: one product with a matrix-free operator that fits in
        # L2 (XXZ L=16, half filling, 12,870 states), where launches and latency
        # count
        dict(_case("product", "xxz", 16, nup=8, columns=1), name="mul_chain_L16"),
        # the reason for a matrix-free operator: one product in the largest
        # sector of the J1-J2 chain (L=32, zero momentum, even parity and flip,
        # 4,707,969 states)
        dict(_case("product", "j1j2", 32, nup=16, k=0, p=1, z=1, columns=1), name="mul_sector_L32"),
        # a momentum sector with complex characters on an odd chain (208,012
        # states, complex vectors), matrix-free
        dict(_case("product", "j1j2", 25, nup=12, k=3, dtype="complex128", columns=1), name="mul_momentum_L25"),
        # a whole particle-number sector without spatial symmetry (40,116,600
        # states), matrix-free: too large to be assembled by habit
        dict(_case("product", "xxz", 28, nup=14, columns=1), name="mul_chain_L28"),
        # the headline product: the assembled Hamiltonian of the L=32 sector
        dict(_case("product", "j1j2", 32, nup=16, k=0, p=1, z=1, form="hamiltonian", columns=1), name="ham_sector_L32"),
        # assembled, complex matrix and vectors: one momentum of a band scan
        dict(_case("product", "j1j2", 26, nup=13, k=5, form="hamiltonian", dtype="complex128", columns=1),
             name="ham_momentum_L26"),
        # assembled, single precision, a model without a particle number: the
        # transverse-field Ising chain (4.8 M states)
        dict(_case("product", "tfim", 28, k=0, p=1, form="hamiltonian", dtype="float32", columns=1),
             name="ham_tfim_L28_f32"),
        # a block of vectors (a filter or a block method) through one call
        dict(_case("product", "j1j2", 28, nup=14, k=0, p=1, form="hamiltonian", columns=8), name="ham_block_L28"),
        # a new sector from nothing: enumerate the basis, assemble the
        # Hamiltonian and apply it once to a host vector, as every program does
        # on its way to its first number
        dict(_case("new_sector", "j1j2", 30, nup=15, k=0, p=1, form="hamiltonian"), name="new_sector_L30"),
        # a small solve, where latency counts: the ground state of the XXZ chain
        # of 12,870 states from a matrix-free operator, value and vector
        dict(_case("eigsh", "xxz", 16, nup=8), name="eigsh_chain_L16"),
        # an ordinary solve: the ground state of a symmetry sector (L=28,
        # 360,000 states) of the assembled Hamiltonian, away from the
        # Majumdar-Ghosh point J2 = 0.5
        dict(_case("eigsh", "j1j2", 28, nup=14, k=0, p=1, z=1, form="hamiltonian", coupling=0.4),
             name="eigsh_sector_L28"),
        # real-time evolution after a quench: ten times of one start state in
        # the zero-momentum, even sector of the Ising chain (L=22, 96,000 states)
        dict(_case("evolve", "tfim", 22, k=0, p=1, form="hamiltonian", dtype="complex128", times=10, t=2.0),
             name="evolve_tfim_L22"),
    ]


def draw(rng):
    coupling = round(rng.uniform(0.2, 0.45), 4)
    kind = rng.choice(["product"] * 6 + ["new_sector", "eigsh", "eigsh", "evolve"])
    if kind == "evolve":
        return _case("evolve", "tfim", rng.randint(10, 22), k=0, p=rng.choice([1, -1]), form="hamiltonian",
                     coupling=2 * coupling, dtype="complex128", times=rng.randint(1, 10),
                     t=round(rng.uniform(0.5, 2.0), 3))
    if kind == "eigsh":
        form = rng.choice(["linear_operator", "hamiltonian"])
        if rng.random() < 0.4:
            L = rng.randint(10, 17)
            return _case("eigsh", "xxz", 2 * (L // 2), nup=L // 2, form=form, coupling=coupling)
        L = 2 * rng.randint(7, 14)
        return _case("eigsh", "j1j2", L, nup=L // 2, k=0, p=1, z=1, form=form, coupling=coupling)
    if kind == "new_sector":
        L = rng.randint(14, 29)
        return _case("new_sector", "j1j2", L, nup=L // 2, k=0, p=rng.choice([1, -1]), form="hamiltonian",
                     coupling=coupling)
    form = rng.choice(["linear_operator", "hamiltonian"])
    columns = rng.choice([1, 1, 1, 2, 5, 8]) if form == "hamiltonian" else 1
    sector = rng.choice(["none", "momentum", "even", "flip", "ising"])
    if sector == "none":
        L = rng.randint(10, 26 if form == "hamiltonian" else 28)
        return _case("product", "xxz", L, nup=L // 2 - rng.randint(0, 2), form=form,
                     coupling=coupling, dtype=rng.choice(["float64", "float32"]), columns=columns if L < 25 else 1)
    if sector == "momentum":
        L = rng.randint(12, 27)
        return _case("product", "j1j2", L, nup=L // 2, k=rng.randint(1, (L - 1) // 2), form=form,
                     coupling=coupling, dtype=rng.choice(["complex128", "complex64"]), columns=columns if L < 25 else 1)
    if sector == "even":
        L = rng.randint(12, 29)
        return _case("product", "j1j2", L, nup=L // 2, k=0, p=rng.choice([1, -1]), form=form,
                     coupling=coupling, dtype=rng.choice(["float64", "float32"]), columns=columns)
    if sector == "flip":
        L = 2 * rng.randint(6, 15)
        return _case("product", "j1j2", L, nup=L // 2, k=0, p=1, z=1, form=form,
                     coupling=coupling, dtype=rng.choice(["float64", "float64", "float32"]), columns=columns)
    L = rng.randint(12, 27)
    return _case("product", "tfim", L, k=0, p=1, form=form, coupling=2 * coupling,
                 dtype=rng.choice(["float64", "float32"]), columns=columns if L < 26 else 1)


# ------------------------------------------------------------------ the models
def _terms(case):
    """Operator terms as (string, [(coefficient, one-based sites...)])."""
    L, model, c = case["L"], case["model"], case["coupling"]
    near = [(i, i % L + 1) for i in range(1, L + 1)]
    if model == "tfim":
        return [("zz", [(1.0, a, b) for a, b in near]), ("x", [(c, i) for i in range(1, L + 1)])]
    if model == "xxz":
        flip, diag = [(0.5, a, b) for a, b in near], [(c, a, b) for a, b in near]
    else:
        far = [(i, (i + 1) % L + 1) for i in range(1, L + 1)]
        flip = [(0.5, a, b) for a, b in near] + [(c / 2, a, b) for a, b in far]
        diag = [(1.0, a, b) for a, b in near] + [(c, a, b) for a, b in far]
    return [("+-", flip), ("-+", flip), ("zz", diag)]


def _parents(case):
    return math.comb(case["L"], case["nup"]) if case["nup"] >= 0 else 2 ** case["L"]


def _rows(case):
    """States of the sector, to the few orbits with a stabiliser."""
    group = (case["L"] if case["k"] >= 0 else 1) * (2 if case["p"] else 1) * (2 if case["z"] else 1)
    return max(1, _parents(case) // group)


def _transitions(case):
    """Off-diagonal elements per row, on average."""
    L, nup = case["L"], case["nup"]
    if case["model"] == "tfim":
        return float(L)
    return (1 if case["model"] == "xxz" else 2) * L * 2.0 * nup * (L - nup) / (L * (L - 1))


def work(case):
    n, hops = _rows(case), _transitions(case)
    size = {"float64": 8, "float32": 4, "complex128": 16, "complex64": 8}[case["dtype"]]
    per_hop = 2 if case["dtype"].startswith("float") else (8 if case["k"] > 0 else 4)
    assembled = 4 * hops + 4          # a packed word per element, its row's length and normalisation
    symmetric = case["k"] >= 0
    if case["kind"] == "product":
        c = case["columns"]
        operator = assembled + 8 if case["form"] == "hamiltonian" else (6 if symmetric else 0)
        return {"bytes": n * (operator + 2 * c * size), "flops": n * hops * per_hop * c}
    if case["kind"] == "new_sector":
        return {"bytes": n * (2 * assembled + 6 + 2 * size), "flops": n * hops * per_hop}
    if case["kind"] == "eigsh":
        step = assembled + 8 + 8 * (_SOLVE_BASIS * 3 // 4 + 2)
        return {"bytes": n * step * _SOLVE_PRODUCTS, "flops": n * _SOLVE_PRODUCTS * (2 * hops + 4 * _SOLVE_BASIS)}
    step = assembled + 8 + 16 * 4
    return {"bytes": n * (step * 30 + 16 * 31 * case["times"]), "flops": n * 30 * (4 * hops + 16 + 8 * case["times"])}


# ------------------------------------------------------------------ prepare and run
def _basis(qs, case):
    kw = {}
    if case["k"] >= 0:
        kw["kblock"] = case["k"]
    if case["p"]:
        kw["pblock"] = case["p"]
    if case["z"]:
        kw["zblock"] = case["z"]
    return qs.SpinBasis1D(case["L"], nup=case["nup"] if case["nup"] >= 0 else None, pauli=case["model"] == "tfim", **kw)


def _operator(qs, case, basis):
    make = qs.Hamiltonian if case["form"] == "hamiltonian" else qs.QuantumLinearOperator
    return make(basis, [qs.OperatorTerm(op, couplings) for op, couplings in _terms(case)])


def _vector(case, seed, n, columns=1):
    """Normal entries, (columns, n), of the case's dtype."""
    g = torch.Generator().manual_seed(1000003 * int(seed) + 7)
    dt = getattr(torch, case["dtype"])
    v = torch.empty((columns, n), dtype=dt)
    real = torch.view_as_real(v) if dt.is_complex else v
    real.copy_(torch.randn(real.shape, generator=g, dtype=real.dtype))
    return v


def _device_vector(case, seed, n, columns=1):
    """The same kind of entries generated on the device."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 7)
    dt = getattr(torch, case["dtype"])
    v = torch.empty((columns, n), dtype=dt, device="cuda")
    (torch.view_as_real(v) if dt.is_complex else v).normal_(generator=g)
    return v


def prepare(case, seed):
    import qsgpu as qs
    from qsgpu import _lib

    s = {"case": case, "qs": qs}
    if case["kind"] == "new_sector":
        # the vector's length is known to such a program once it has the basis
        n = _basis(qs, case).Ns
        s["x"] = _vector(case, seed, n)[0].numpy()
        return s
    s["basis"] = _basis(qs, case)
    s["op"] = _operator(qs, case, s["basis"])
    n = s["basis"].Ns
    if case["kind"] == "eigsh":
        s["v0"] = _vector(case, seed, n)[0].numpy()
    elif case["kind"] == "evolve":
        v = _vector(case, seed, n)[0].numpy()
        s["v0"] = v / np.linalg.norm(v)
        s["times"] = _times(case)
    else:
        # vectors on the device: the products are ordered on the program's stream
        s["x"] = _device_vector(case, seed, n, case["columns"])
        s["y"] = torch.zeros_like(s["x"])
        s["stream"] = torch.cuda.Stream()
        lib = _lib.load()
        _lib.check(lib.qs_op_set_stream(s["op"]._h, ctypes.c_void_p(s["stream"].cuda_stream)))
        code = {"float64": _lib.QS_F64, "float32": _lib.QS_F32, "complex128": _lib.QS_C128,
                "complex64": _lib.QS_C64}[case["dtype"]]
        one, zero = np.array([1.0, 0.0]), np.array([0.0, 0.0])
        s["keep"] = (one, zero)
        s["call"] = (lib.qs_op_matvec, _lib.check,
                     (s["op"]._h, 0, _lib.ptr(one), ctypes.c_void_p(s["x"].data_ptr()), code, _lib.ptr(zero),
                      ctypes.c_void_p(s["y"].data_ptr()), code, case["columns"], _lib.QS_MEM_DEVICE))
        torch.cuda.synchronize()
    return s


def _times(case):
    return np.linspace(case["t"] / case["times"], case["t"], case["times"])


def run(state):
    case, qs = state["case"], state["qs"]
    if case["kind"] == "product":
        matvec, check, args = state["call"]
        check(matvec(*args))
        return state["y"]
    if case["kind"] == "new_sector":
        H = _operator(qs, case, _basis(qs, case))
        return H.dot(state["x"])
    if case["kind"] == "eigsh":
        values, vectors = qs.eigsh(state["op"], k=1, which="SA", tol=1e-12, v0=state["v0"])
        return [values, vectors]
    return qs.evolve(state["op"], state["v0"], 0.0, state["times"])


# ------------------------------------------------------------------ 64-bit results
def _where():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _states(L, nup, dev):
    """Ascending states of L sites: all, or those with nup set bits."""
    if nup < 0:
        return torch.arange(2 ** L, dtype=torch.int64, device=dev)
    # bits 0 .. l-1 with each weight that a state of weight nup can have there
    rows = {0: torch.zeros(1, dtype=torch.int64, device=dev)}
    for l in range(1, L + 1):
        new = {}
        for w in range(max(0, nup - (L - l)), min(nup, l) + 1):
            parts = ([rows[w]] if w in rows else []) + ([rows[w - 1] | (1 << (l - 1))] if w - 1 in rows else [])
            new[w] = torch.cat(parts)
        rows = new
    return rows[nup]


def _images(case, s):
    """(image, its element's character) of s under every element of the sector's group."""
    L = case["L"]
    full = (1 << L) - 1
    bases = [(s, 1.0)]
    if case["p"]:
        r = torch.zeros_like(s)
        for i in range(L):
            r |= ((s >> i) & 1) << (L - 1 - i)
        bases.append((r, float(case["p"])))
    if case["z"]:
        bases += [(b ^ full, c * case["z"]) for b, c in bases]
    for b, c in bases:
        for j in range(L if case["k"] >= 0 else 1):
            phase = np.exp(2j * np.pi * case["k"] * j / L) if case["k"] > 0 else 1.0
            yield (b if j == 0 else ((b << j) | (b >> (L - j))) & full), c * phase


class _Sector:
    """The sector's representatives, diagonal and transitions, from scratch."""

    def __init__(self, case, dev):
        self.case, self.dev = case, dev
        self.symmetric = case["k"] >= 0 or case["p"] != 0 or case["z"] != 0
        self.complex = case["k"] > 0 and 2 * case["k"] != case["L"]
        parents = _states(case["L"], case["nup"], dev)
        if not self.symmetric:
            self.reps, self.stab = parents, None
        else:
            kept = []
            for part in torch.split(parents, 1 << 26):
                for i, (t, _) in enumerate(_images(case, part)):
                    if i == 0:
                        alive = torch.ones(part.shape, dtype=torch.bool, device=dev)
                    alive &= t >= part
                kept.append(part[alive])
            reps = torch.cat(kept)
            del parents, kept
            weight = torch.zeros(reps.shape, dtype=torch.complex128, device=dev)
            stab = torch.zeros(reps.shape, dtype=torch.int64, device=dev)
            for t, c in _images(case, reps):
                same = t == reps
                weight += same * complex(c)
                stab += same
            keep = weight.abs() > 0.5
            self.reps, self.stab = reps[keep], stab[keep].double()
        self.n = self.reps.numel()
        zs = 1.0 if case["model"] == "tfim" else 0.5
        self.diag = torch.zeros(self.n, dtype=torch.float64, device=dev)
        self.moves = {}
        for op, couplings in _terms(case):
            for c in couplings:
                sites = [q - 1 for q in c[1:]]
                if op == "zz":
                    odd = ((self.reps >> sites[0]) ^ (self.reps >> sites[1])) & 1
                    self.diag += c[0] * zs * zs * (1 - 2 * odd).double()
                elif op == "x":
                    self.moves[(1 << sites[0], None)] = self.moves.get((1 << sites[0], None), 0.0) + c[0]
                elif op == "+-":   # with its "-+" of the same bond: an exchange of two unequal spins
                    key = ((1 << sites[0]) | (1 << sites[1]), (sites[0], sites[1]))
                    self.moves[key] = self.moves.get(key, 0.0) + c[0]

    def hops(self):
        """(columns, values) of one transition of every row, for each transition."""
        for (mask, bond), amplitude in self.moves.items():
            t = self.reps ^ mask
            w = torch.full((self.n,), amplitude, dtype=torch.complex128 if self.complex else torch.float64,
                           device=self.dev)
            if bond is not None:
                w = w * (((self.reps >> bond[0]) ^ (self.reps >> bond[1])) & 1)
                t = torch.where(w != 0, t, self.reps)
            if self.symmetric:
                chars, best, at = [], t.clone(), torch.zeros(t.shape, dtype=torch.int64, device=self.dev)
                for i, (u, c) in enumerate(_images(self.case, t)):
                    chars.append(complex(c))
                    less = u < best
                    best = torch.where(less, u, best)
                    at = torch.where(less, torch.full_like(at, i), at)
                chi = torch.tensor(chars, dtype=torch.complex128, device=self.dev)
                chi = chi if self.complex else chi.real.contiguous()
                col = torch.searchsorted(self.reps, best).clamp_(max=self.n - 1)
                w = w * (self.reps[col] == best) * chi[at] * torch.sqrt(self.stab[col] / self.stab)
            else:
                col = torch.searchsorted(self.reps, t)
            yield col, w

    def apply(self, x, transitions=None):
        """H x for rows of x (..., n)."""
        y = self.diag * x
        for col, w in transitions if transitions is not None else self.hops():
            y = y + w * x[..., col]
        return y


def _lowest(matvec, v, most=400):
    """The lowest eigenvalue by Lanczos with full reorthogonalisation."""
    V = [v / torch.linalg.vector_norm(v)]
    a, b, last = [], [], None
    for j in range(min(most, v.numel())):
        w = matvec(V[-1])
        a.append(float(torch.vdot(V[-1], w).real))
        Q = torch.stack(V)
        for _ in range(2):
            w = w - (Q.conj() @ w) @ Q
        beta = float(torch.linalg.vector_norm(w))
        if j % 10 == 9 or beta < 1e-13:
            T = np.diag(a) + np.diag(b, 1) + np.diag(b, -1)
            e, U = np.linalg.eigh(T)
            last = e[0]
            if abs(beta * U[-1, 0]) < 1e-12:
                break
        b.append(beta)
        V.append(w / beta)
    return last


def _propagate(matvec, radius, v, times):
    """exp(-i H t) v at every time by one Chebyshev expansion on [-radius, radius]."""
    m = int(radius * max(times) * 1.2) + 60
    theta = 2 * np.pi * np.arange(4 * m) / (4 * m)
    coef = []
    for t in times:   # exp(-i z cos(theta)) = c_0 + 2 sum_k c_k cos(k theta)
        c = np.fft.fft(np.exp(-1j * radius * t * np.cos(theta)))[:m] / (4 * m)
        c[1:] *= 2
        coef.append(c)
    out = [coef[i][0] * v for i in range(len(times))]
    prev, cur = v, matvec(v) / radius
    for q in range(1, m):
        for i in range(len(times)):
            if abs(coef[i][q]) > 1e-18:
                out[i] = out[i] + complex(coef[i][q]) * cur
        prev, cur = cur, 2 * matvec(cur) / radius - prev
    return torch.stack(out, dim=1)


def exact(case, seed):
    dev = _where()
    sector = _Sector(case, dev)
    n = sector.n
    if case["kind"] == "product":
        if dev.type == "cuda":
            x = _device_vector(case, seed, n, case["columns"])
        else:
            x = _vector(case, seed, n, case["columns"])
        x = x.to(torch.complex128 if x.is_complex() else torch.float64)
        if case["columns"] * n > 1 << 26:   # column by column where all at once would be large
            return torch.stack([sector.apply(c) for c in x])
        return sector.apply(x)
    if case["kind"] == "new_sector":
        return sector.apply(_vector(case, seed, n)[0].to(dev))
    transitions = list(sector.hops())
    v = _vector(case, seed, n)[0].to(dev)
    if case["kind"] == "eigsh":
        # the vector's sign is the solver's own
        return [np.array([_lowest(lambda u: sector.apply(u, transitions), v)]), None]
    radius = 1.02 * float(sector.diag.abs().max() + sum(abs(a) for a in sector.moves.values()))
    v = v / torch.linalg.vector_norm(v)
    return _propagate(lambda u: sector.apply(u, transitions), radius, v, _times(case))
