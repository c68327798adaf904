"""Benchmark of the hot path: the symmetry-reduced Hamiltonian action H.v and the
Lanczos ground-state solve that consumes it, on one GPU per process.

Default workload: Heisenberg J1-J2 chain L=32, nup=16, kblock=0, pblock=+1,
zblock=+1 (N = 4,707,969 representatives), J1=1.0, J2=0.5, FP64.

A step is one matvec y = H x over the whole sector.  `value` is the H.v
throughput in GB/s of algorithmic traffic (bytes per row defined below) with x, y
resident in HBM; `e2e` is the same metric through the C ABI with host buffers
(host->device copy of x and device->host copy of y inside every timed step).
Lanczos solves/s (eigsh k=1 :SA, tol 1e-10), the FP32, double-float and
fixed-point forms are reported beside it, and side workloads under
`workloads` (XXZ L=16, batched sectors, TFIM evolve, FTLM, block tools,
SpinBasisGeneral, the XXZ roofline sweep L=24..30, serving; `--no-sections`
skips them, `--only-section KEY` runs one).  Synthetic data only (seeded
N(0,1) vectors; the Hamiltonian is the model itself).  N > 1 runs
independent replicas (the path is not sharded).

`--impl reference` times the CPU restatement of the reference's algorithm
(oracle/, representative-space port, all host threads) on a bounded sample of
rows of the same workload and prints the same metric.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
for _p in (os.path.join(ROOT, "quspin.jl_gb300"), os.path.join(ROOT, "oracle")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

METRIC = "H·v GB/s (% HBM peak), Lanczos solves/s, p50/p99 latency; FP32 vs FP64 form"


def load_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def j1j2_spec(L, J1=1.0, J2=0.5):
    b1 = [(i, i % L + 1) for i in range(1, L + 1)]
    b2 = [(i, (i + 1) % L + 1) for i in range(1, L + 1)]
    return [("+-", [(J1 / 2, a, b) for a, b in b1] + [(J2 / 2, a, b) for a, b in b2]),
            ("-+", [(J1 / 2, a, b) for a, b in b1] + [(J2 / 2, a, b) for a, b in b2]),
            ("zz", [(J1, a, b) for a, b in b1] + [(J2, a, b) for a, b in b2])]


WORKLOADS = {
    # traffic: dram bytes read + written by one launch of the FP64 sliced-ELL
    # product on this workload, from an ncu capture of
    # `bench.py --profile-range product64` on a GB300 (not measured in the
    # timed run; traffic_source names the summary it comes from)
    "j1j2_L32_k0_p1_z1": dict(L=32, nup=16, sym=dict(kblock=0, pblock=1, zblock=1), J2=0.5,
                              desc="Heisenberg J1-J2 chain L=32, nup=16, kblock=0, pblock=+1, zblock=+1, "
                                   "J1=1.0, J2=0.5", traffic=788.81e6 + 27.69e6,
                              traffic_source="ncu dram__bytes_read.sum + dram__bytes_write.sum of one launch, "
                                             "profiles/sell_fp64_j1j2_L32_k0p1z1.md (not measured in this run)"),
    "j1j2_L24_k0_p1_z1": dict(L=24, nup=12, sym=dict(kblock=0, pblock=1, zblock=1), J2=0.5,
                              desc="Heisenberg J1-J2 chain L=24, nup=12, kblock=0, pblock=+1, zblock=+1 (small case)"),
}


def alive_transitions(states, L, J2):
    """Average number of off-diagonal transitions that survive per row: one per
    bond whose two spins differ (the +- / -+ pair), J1 and J2 bonds."""
    s = states.astype(np.uint64)
    tot = np.zeros(s.size)
    for d in (1, 2) if J2 else (1,):
        for i in range(L):
            j = (i + d) % L
            tot += (((s >> np.uint64(i)) ^ (s >> np.uint64(j))) & np.uint64(1)).astype(np.float64)
    return float(tot.mean())


def asm_bytes_per_row(nbar, vec_bytes=8):
    """Compulsory HBM bytes per row of one product with the assembled operator:
    4 bytes per stored transition (packed column + value code), a 2-byte row
    length, the 2-byte stabiliser code, the diagonal, x[r] and the y[r] write.
    The x gathers of the transitions hit L2 when x fits in it and are not
    counted."""
    return 4 * nbar + 2 + 2 + 3 * vec_bytes


class ClockSampler:
    def __init__(self):
        self.rows = []
        self.proc = None
        self.thread = None

    def start(self):
        cmd = ["nvidia-smi", "--query-gpu=index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
               "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
               "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap",
               "--format=csv,noheader,nounits", "-lms", "200"]
        dev = os.environ.get("CUDA_VISIBLE_DEVICES", "").split(",")[0]
        if dev:
            cmd += ["-i", dev]
        try:
            self.proc = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
            return

        def rd():
            for line in self.proc.stdout:
                self.rows.append([x.strip() for x in line.split(",")])
        self.thread = threading.Thread(target=rd, daemon=True)
        self.thread.start()

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        if self.thread:
            self.thread.join(timeout=2)
        sm = [float(r[1]) for r in self.rows if len(r) >= 9 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) >= 9 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in self.rows:
            if len(r) >= 9:
                for k, name in enumerate(names):
                    if r[5 + k].lower().startswith("active"):
                        reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(self.rows)}


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        backend = "nccl" if os.environ.get("QS_BENCH_BACKEND", "nccl") == "nccl" else "gloo"
        dist.init_process_group(backend=backend)
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(world, v, device=None):
    if world == 1:
        return v
    import torch
    import torch.distributed as dist
    t = torch.tensor([v], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_value(world, bytes_per_step, t_step):
    """Whole-job GB/s of `world` independent replicas: every replica moves
    bytes_per_step per step, and the slowest replica's step time counts."""
    return world * bytes_per_step / t_step / 1e9


def cpu_port_sample(wl, nthreads, target_s=10.0, seed=20261203):
    """Times the oracle's representative-space port on contiguous row samples
    until ~target_s of CPU work; returns (seconds per row, rows timed, nbar, N)."""
    import oracle
    L, nup = wl["L"], wl["nup"]
    rb = oracle.RepBasis(L, nup=nup, pauli=False, nthreads=nthreads, **wl["sym"])
    spec = j1j2_spec(L, 1.0, wl["J2"])
    pk = oracle.pack_terms(spec)
    n = rb.Ns
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n).astype(np.complex128)
    d = rb.diagonal(spec)
    rows_done, t_total = 0, 0.0
    block = max(1024, n // 256)
    start = n // 3
    while t_total < target_s and rows_done < n:
        r0 = (start + rows_done) % n
        r1 = min(n, r0 + block)
        t = time.perf_counter()
        rb.matvec(spec, x, diag=d, rows=(r0, r1), packed=pk)
        t_total += time.perf_counter() - t
        rows_done += r1 - r0
        block = min(n, block * 2)
    nbar = alive_transitions(rb.states[n // 3: n // 3 + 100000], L, wl["J2"])
    return t_total / rows_done, rows_done, nbar, n, t_total


REF_BLOCKS = 16   # a reference-arm step is 1/16 of the sector's rows


def run_reference(args, wl, world, rank):
    """The reference arm: the oracle's representative-space restatement of the
    reference matvec on all host cores, on the same workload and metric.  One
    step is one contiguous block of 1/REF_BLOCKS of the sector's rows (the
    blocks rotate through the sector, so REF_BLOCKS steps make one whole
    product); every step is timed as it runs, nothing is extrapolated, and the
    GB/s counts the bytes of the rows each step computed (4 per transition +
    28 per row, the GPU arm's byte model, with the sector's exact transition
    count)."""
    if rank != 0:
        return
    import oracle
    oracle.lib()
    nthreads = os.cpu_count() or 1
    L, nup = wl["L"], wl["nup"]
    rb = oracle.RepBasis(L, nup=nup, pauli=False, nthreads=nthreads, **wl["sym"])
    spec = j1j2_spec(L, 1.0, wl["J2"])
    pk = oracle.pack_terms(spec)
    n = rb.Ns
    x = np.random.default_rng(20261203).standard_normal(n).astype(np.complex128)
    d = rb.diagonal(spec)
    nbar = alive_transitions(rb.states, L, wl["J2"])
    bounds = [(n * i // REF_BLOCKS, n * (i + 1) // REF_BLOCKS) for i in range(REF_BLOCKS)]
    for i in range(args.warmup):
        rb.matvec(spec, x, diag=d, rows=bounds[i % REF_BLOCKS], packed=pk)
    dts, rows = [], 0
    for i in range(args.steps):
        r0, r1 = bounds[i % REF_BLOCKS]
        t = time.perf_counter()
        rb.matvec(spec, x, diag=d, rows=(r0, r1), packed=pk)
        dts.append(time.perf_counter() - t)
        rows += r1 - r0
    # the port computes in complex128; the metric counts the FP64 real form's bytes
    gbs = asm_bytes_per_row(nbar, 8) * rows / sum(dts) / 1e9
    line = {
        "metric": METRIC, "value": gbs, "unit": "GB/s", "impl": "reference", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": float(np.mean(dts)) * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": wl["desc"], "N": n, "nnz": int(round(nbar * n)),
                   "step": f"H.v over one block of {REF_BLOCKS} equal row blocks of the sector (blocks rotate; "
                           f"{REF_BLOCKS} steps = one whole product)"},
        "cpu_baseline": {"value": gbs, "unit": "GB/s", "cores": nthreads, "kind": "port",
                         "sample": f"{args.steps} steps of {n // REF_BLOCKS} rows each ({sum(dts):.1f} s), "
                                   "representative-space restatement of the reference matvec on all host cores "
                                   "(the reference's own projector algorithm needs the 601M-state parent sector)"},
        "e2e": {"value": gbs, "unit": "GB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def xxz_spec(L, J=1.0, delta=0.5):
    bonds = [(i, i % L + 1) for i in range(1, L + 1)]
    return [("+-", [(J / 2, a, b) for a, b in bonds]), ("-+", [(J / 2, a, b) for a, b in bonds]),
            ("zz", [(J * delta, a, b) for a, b in bonds])]


def tfim_spec(L, J=1.0, h=0.7):
    bonds = [(i, i % L + 1) for i in range(1, L + 1)]
    return [("zz", [(J, a, b) for a, b in bonds]), ("x", [(h, i) for i in range(1, L + 1)])]


def section_c1(qs, torch, timed_events):
    """Periodic XXZ L=16, nup=8 (12,870 states), no spatial symmetry, FP64:
    one QuantumLinearOperator matvec and eigsh k=4 :SA (tol 1e-10, v0 = ones;
    warm, best of 3: the solver assembles the operator for each call),
    against the oracle's restatement of the reference algorithm (serial scatter
    with per-state lookups, 1 thread) and SciPy's ARPACK over it, and the
    matvec of the representative-space port on all host cores."""
    import oracle
    L = 16
    spec = xxz_spec(L)
    b = qs.SpinBasis1D(L, nup=8, pauli=False)
    op = qs.QuantumLinearOperator(b, [qs.OperatorTerm(o, c) for o, c in spec])
    n = b.Ns
    x = np.random.default_rng(20261203).standard_normal(n)
    us = timed_events(op, x, 200) * 1e3
    v0 = np.ones(n) / np.sqrt(n)
    # warm (the first call also builds the per-device kernel attributes), best of 3
    vals = qs.eigsh(op, k=4, which="SA", tol=1e-10, v0=v0, return_eigenvectors=False)
    t_gpu = 1e30
    for _ in range(3):
        torch.cuda.synchronize()
        t = time.perf_counter()
        vals = qs.eigsh(op, k=4, which="SA", tol=1e-10, v0=v0, return_eigenvectors=False)
        torch.cuda.synchronize()
        t_gpu = min(t_gpu, time.perf_counter() - t)
    ref = oracle.RefBasis(L, nup=8, pauli=False)
    ct = oracle.consolidate_terms(spec)
    d = ref.extract_diagonal(ct)
    pk = oracle.pack_terms(ct)
    t = time.perf_counter()
    reps = 20
    for _ in range(reps):
        ref.qlo_matvec(ct, x, total_diag=d, packed=pk)
    cpu_mv = (time.perf_counter() - t) / reps
    t = time.perf_counter()
    cvals, _ = oracle.eigsh_arpack(lambda v: ref.qlo_matvec(ct, v, total_diag=d, packed=pk).real, n, 4,
                                   np.float64, v0=v0, tol=1e-10)
    t_cpu = time.perf_counter() - t
    # the representative-space port on all host cores (no symmetry here: the parent sector)
    ncores = os.cpu_count() or 1
    rb = oracle.RepBasis(L, nup=8, pauli=False, nthreads=ncores)
    dr = rb.diagonal(spec)
    pkr = oracle.pack_terms(spec)
    rb.matvec(spec, x.astype(np.complex128), diag=dr, packed=pkr)
    t = time.perf_counter()
    for _ in range(reps):
        rb.matvec(spec, x.astype(np.complex128), diag=dr, packed=pkr)
    cpu_mv_all = (time.perf_counter() - t) / reps
    return {"workload": "periodic XXZ L=16, nup=8, J=1, Delta=0.5, pauli=false, N=12870",
            "matvec_us_gpu": us, "matvec_us_cpu_reference_algorithm": cpu_mv * 1e6,
            "matvec_us_cpu_port_all_cores": cpu_mv_all * 1e6, "cpu_port_cores": ncores,
            "eigsh_k4_s_gpu": t_gpu, "eigsh_k4_s_cpu_arpack_reference_algorithm": t_cpu,
            "eigenvalues": [float(v) for v in vals],
            "max_abs_diff_vs_cpu": float(np.max(np.abs(np.sort(vals) - np.sort(cvals)))),
            "cpu_cores": 1}


def tfim_product_state(qs, b, L, seed=20261203):
    """The homogeneous product state (cos th |dn> + e^{i ph} sin th |up>)^L
    expressed in the sector's columns (th, ph seeded), normalised."""
    rng = np.random.default_rng(seed)
    th, ph = rng.uniform(0, np.pi), rng.uniform(0, 2 * np.pi)
    reps = b.orbit_minima()
    pop = np.zeros(reps.size, dtype=np.int64)
    for i in range(L):
        pop += ((reps >> np.uint64(i)) & np.uint64(1)).astype(np.int64)
    orb = b.group_order / b.stabilizers().astype(np.float64)
    up, dn = np.exp(1j * ph) * np.sin(th), np.cos(th)
    v0 = (up ** pop) * (dn ** (L - pop)) * np.sqrt(orb)
    return v0 / np.linalg.norm(v0)


def section_c3(qs, torch, n_times=50, fp32_times=10, cpu_L=24, cpu_times=5):
    """TFIM L=30 periodic, J=1, h=0.7 (pauli), k=0, p=+1, no U(1) (N=17,920,860):
    evolve ComplexF64 from the homogeneous product state to the 50 times
    range(0.1, 5.0) (krylov_dim 30, tol 1e-9): one evolve call over all times
    (the reference's _krylov_expmv_times, failing times re-run concurrently)
    in FP64 and in the double-float form, the FP32 form on the first
    `fp32_times`, and all 50 times stepwise (from each time to the next) in
    FP64 and double-float; states compared where they overlap.  CPU baseline:
    the oracle's restatement of _krylov_expmv_times over the representative-
    space product on all host cores, at L=`cpu_L` on the first `cpu_times`
    times (the L=30 product alone takes tens of seconds on the host), with the
    GPU's FP64 evolve of the same input beside it."""
    L = 30
    b = qs.SpinBasis1D(L, pauli=True, kblock=0, pblock=1)
    t = time.perf_counter()
    H = qs.Hamiltonian(b, [qs.OperatorTerm(o, c) for o, c in tfim_spec(L)])
    t_asm = time.perf_counter() - t
    v0 = tfim_product_state(qs, b, L)
    times = np.linspace(0.1, 5.0, 50)[:n_times]
    out = {"workload": "TFIM L=30, J=1, h=0.7, k=0, p=+1, N=%d, nnz=%d, %d times to t=%.1f" % (
        b.Ns, H.nnz, times.size, times[-1]), "assemble_s": t_asm}
    res = {}
    for prec, nt in (("fp64df", times.size), ("fp64", times.size), ("fp32", min(fp32_times, times.size))):
        torch.cuda.synchronize()
        t = time.perf_counter()
        st = qs.evolve(H, v0, 0.0, times[:nt], tol=1e-9, krylov_dim=30, precision=prec)
        out[f"evolve_s_{prec}"] = time.perf_counter() - t
        out[f"times_{prec}"] = int(nt)
        res[prec] = st
        out[f"norm_drift_{prec}"] = float(np.max(np.abs(np.linalg.norm(st, axis=0) - 1)))
    out["evolves_per_s_fp64"] = 1.0 / out["evolve_s_fp64"]
    out["evolves_per_s_fp64df"] = 1.0 / out["evolve_s_fp64df"]
    out["fp64df_speedup_vs_fp64"] = out["evolve_s_fp64"] / out["evolve_s_fp64df"]
    # the same 50 times from each to the next (evolve(..., stepwise=True)), FP64
    # and double-float, against the reference-faithful FP64 states
    for prec in ("fp64", "fp64df"):
        torch.cuda.synchronize()
        t = time.perf_counter()
        sw = qs.evolve(H, v0, 0.0, times, tol=1e-9, krylov_dim=30, precision=prec, stepwise=True)
        out[f"evolve_s_{prec}_stepwise"] = time.perf_counter() - t
        out[f"{prec}_stepwise_vs_fp64_state_err"] = float(np.max(np.linalg.norm(sw - res["fp64"], axis=0)))
    out["fp64df_vs_fp64_state_err"] = float(np.max(np.linalg.norm(res["fp64df"] - res["fp64"], axis=0)))
    nt32 = res["fp32"].shape[1]
    err32 = float(np.max(np.linalg.norm(res["fp32"] - res["fp64"][:, :nt32], axis=0)))
    out["fp32_vs_fp64_state_err"] = err32
    out["fp32_meets_state_tol_1e-9"] = bool(err32 <= 1e-9)
    out["note"] = ("FP64 and double-float run all %d times; FP32 runs the first %d and its state error against "
                   "FP64 (%.1e) %s the 1e-9 state target, so the FP32 form of this workload is %s" % (
                       times.size, nt32, err32, "meets" if err32 <= 1e-9 else "misses",
                       "met" if err32 <= 1e-9 else "not met; the double-float form is the fast FP64-class one"))
    del H
    # CPU baseline at a size the host finishes in tens of seconds, GPU beside it
    try:
        import oracle
        oracle.lib()
        nthreads = os.cpu_count() or 1
        spec = tfim_spec(cpu_L)
        bs = qs.SpinBasis1D(cpu_L, pauli=True, kblock=0, pblock=1)
        Hs = qs.Hamiltonian(bs, [qs.OperatorTerm(o, c) for o, c in spec])
        vs = tfim_product_state(qs, bs, cpu_L)
        ts = times[:cpu_times]
        rb = oracle.RepBasis(cpu_L, pauli=True, nthreads=nthreads, kblock=0, pblock=1)
        pk = oracle.pack_terms(spec)
        d = rb.diagonal(spec)
        count = [0]

        def mv(z):
            count[0] += 1
            return rb.matvec(spec, z, diag=d, packed=pk)
        t = time.perf_counter()
        cst = oracle.krylov_expmv_times(mv, vs, [-1j * x for x in ts], hermitian=True, tol=1e-9, krylov_dim=30)
        t_cpu = time.perf_counter() - t
        qs.evolve(Hs, vs, 0.0, ts, tol=1e-9, krylov_dim=30)   # warm-up
        torch.cuda.synchronize()
        t = time.perf_counter()
        gst = qs.evolve(Hs, vs, 0.0, ts, tol=1e-9, krylov_dim=30)
        t_gpu = time.perf_counter() - t
        out["cpu_baseline"] = {
            "kind": "port", "cores": nthreads, "L": cpu_L, "N": bs.Ns, "times": int(ts.size),
            "cpu_evolve_s": t_cpu, "cpu_products": count[0], "gpu_fp64_evolve_s": t_gpu,
            "gpu_vs_cpu": t_cpu / t_gpu, "max_state_diff": float(np.max(np.linalg.norm(gst - cst, axis=0))),
            "sample": "the oracle's _krylov_expmv_times restatement over the representative-space product on all "
                      "host cores, TFIM L=%d k=0 p=+1, the first %d times; the GPU FP64 evolve of the same "
                      "input beside it" % (cpu_L, ts.size)}
    except Exception as exc:  # the baseline is reported, never required
        out["cpu_baseline"] = {"error": f"{type(exc).__name__}: {exc}"}
    return out


def section_c4(qs, torch):
    """All momentum sectors (p=+-1 at k=0, 13) of the J1-J2 chain L=26, nup=13,
    J2=0.3: ground state of every sector, batched (one launch per Lanczos step
    for all 28 sectors) against sector-by-sector eigsh."""
    L = 26
    spec = j1j2_spec(L, 1.0, 0.3)
    terms = [qs.OperatorTerm(o, c) for o, c in spec]
    syms = []
    for k in range(L):
        if k in (0, L // 2):
            syms += [dict(kblock=k, pblock=1), dict(kblock=k, pblock=-1)]
        else:
            syms.append(dict(kblock=k))
    torch.cuda.synchronize()
    t = time.perf_counter()
    ops = [qs.Hamiltonian(qs.SpinBasis1D(L, nup=13, pauli=False, **sy), terms) for sy in syms]
    t_build = time.perf_counter() - t
    sizes = [o.Ns for o in ops]
    # warm-up: graph capture and the pooled buffers
    t = time.perf_counter()
    for prec in ("fp64", "fp64df", "fp32"):
        qs.eigsh_batch(ops, k=1, tol=1e-10, precision=prec)
    t_warm = time.perf_counter() - t
    timed = {}
    vals = {}
    infos = []
    for prec in ("fp64", "fp64df", "fp32"):
        torch.cuda.synchronize()
        t = time.perf_counter()
        vals[prec] = qs.eigsh_batch(ops, k=1, tol=1e-10, precision=prec, infos=infos if prec == "fp64" else None)[:, 0]
        timed[prec] = time.perf_counter() - t
    # the CPU restatement of the reference matvec on all host cores, timed on a
    # row sample of one k = 1 sector and scaled by the products these solves used
    cpu = None
    try:
        import oracle
        oracle.lib()
        nthreads = os.cpu_count() or 1
        rb = oracle.RepBasis(L, nup=13, pauli=False, nthreads=nthreads, kblock=1)
        x = np.random.default_rng(1).standard_normal(rb.Ns).astype(np.complex128)
        d = rb.diagonal(spec)
        pk = oracle.pack_terms(spec)
        rows, tt, blk = 0, 0.0, 4096
        while tt < 3.0 and rows < rb.Ns:
            r1 = min(rb.Ns, rows + blk)
            t = time.perf_counter()
            rb.matvec(spec, x, diag=d, rows=(rows, r1), packed=pk)
            tt += time.perf_counter() - t
            rows, blk = r1, blk * 2
        row_matvecs = sum(o.Ns * i["matvecs"] for o, i in zip(ops, infos))
        cpu = {"cores": nthreads, "kind": "port", "seconds_per_row": tt / rows,
               "estimated_solves_per_s": len(ops) / (row_matvecs * tt / rows),
               "sample": f"{rows} rows of the k=1 sector; products only (the FP64 batched solves' counts)"}
    except Exception as exc:  # the estimate is reported, never required
        cpu = {"error": f"{type(exc).__name__}: {exc}"}
    # the plain FP64 GPU path: one eigsh per sector
    t = time.perf_counter()
    vs = np.array([qs.eigsh(o, k=1, which="SA", tol=1e-10, return_eigenvectors=False)[0] for o in ops])
    t_seq = time.perf_counter() - t
    scale = float(np.max(np.abs(vs)))
    return {"workload": "J1-J2 L=26, nup=13, J2=0.3, %d sectors, %d states" % (len(ops), sum(sizes)),
            "sector_sizes": [min(sizes), max(sizes)], "build_s": t_build, "warmup_s": t_warm,
            "sequential_fp64_solves_per_s": len(ops) / t_seq,
            "batched_fp64_solves_per_s": len(ops) / timed["fp64"],
            "batched_fp64df_solves_per_s": len(ops) / timed["fp64df"],
            "batched_fp32_polished_solves_per_s": len(ops) / timed["fp32"],
            "batched_fp32_polished_speedup": t_seq / timed["fp32"],
            "max_rel_diff_fp32_batched_vs_sequential": float(np.max(np.abs(vals["fp32"] - vs))) / scale,
            "batched_fp64_speedup": t_seq / timed["fp64"],
            "batched_fp64df_speedup": t_seq / timed["fp64df"],
            "max_rel_diff_fp64_batched_vs_sequential": float(np.max(np.abs(vals["fp64"] - vs))) / scale,
            "max_rel_diff_fp64df_batched_vs_sequential": float(np.max(np.abs(vals["fp64df"] - vs))) / scale,
            "ground_energy": float(np.min(vs)), "cpu_port_estimate": cpu}


def section_ftlm(qs, torch, R=32, m=100, seq_sample=8):
    """Finite-temperature Lanczos on the J1-J2 chain L=26, nup=13, J2=0.3,
    k=0, p=+1: R seeded random start vectors, m Lanczos steps each, the
    energy and nearest-neighbour zz estimates at three temperatures.  The R
    recurrences run in one engine (lanczos_batch) against one lanczos_full
    per vector."""
    L = 26
    spec = j1j2_spec(L, 1.0, 0.3)
    zz = [("zz", [(1.0, i, i % L + 1) for i in range(1, L + 1)])]
    basis = qs.SpinBasis1D(L, nup=13, pauli=False, kblock=0, pblock=1)
    H = qs.Hamiltonian(basis, [qs.OperatorTerm(o, c) for o, c in spec])
    ZZ = qs.Hamiltonian(basis, [qs.OperatorTerm(o, c) for o, c in zz])
    n = H.Ns
    V0 = np.random.default_rng(20261203).standard_normal((R, n)).T   # Ns x R, each start contiguous
    beta = [0.5, 1.0, 2.0]
    obs = {"H": H, "ZZ": ZZ}

    def estimate(samples):
        acc = {"H": 0.0, "ZZ": 0.0, "Z": 0.0}
        for E, V, Q in samples:
            res, ident = qs.ftlm_static_iteration(obs, E, V, Q, beta=beta)
            acc["H"] = acc["H"] + res["H"]
            acc["ZZ"] = acc["ZZ"] + res["ZZ"]
            acc["Z"] = acc["Z"] + ident
        return acc

    estimate(qs.lanczos_batch(H, V0[:, :2], m))   # warm-up: tiles, graph capture
    torch.cuda.synchronize()
    t = time.perf_counter()
    acc = estimate(qs.lanczos_batch(H, V0, m))
    t_batch = time.perf_counter() - t
    t = time.perf_counter()
    acc_seq = estimate([qs.lanczos_full(H, V0[:, r], m) for r in range(seq_sample)])
    t_seq = time.perf_counter() - t
    acc_b8 = estimate(qs.lanczos_batch(H, V0[:, :seq_sample], m))
    energy = (acc["H"] / acc["Z"]).tolist()
    cpu = None
    try:
        import oracle
        oracle.lib()
        nthreads = os.cpu_count() or 1
        rb = oracle.RepBasis(L, nup=13, pauli=False, nthreads=nthreads, kblock=0, pblock=1)
        x = V0[:, 0].astype(np.complex128)
        d = rb.diagonal(spec)
        pk = oracle.pack_terms(spec)
        rows, tt, blk = 0, 0.0, 4096
        while tt < 3.0 and rows < rb.Ns:
            r1 = min(rb.Ns, rows + blk)
            t = time.perf_counter()
            rb.matvec(spec, x, diag=d, rows=(rows, r1), packed=pk)
            tt += time.perf_counter() - t
            rows, blk = r1, blk * 2
        per_sample = (m + 2) * n * tt / rows
        cpu = {"cores": nthreads, "kind": "port", "estimated_samples_per_s": 1.0 / per_sample,
               "sample": f"{rows} rows of the sector; products only (m + 2 per sample)"}
    except Exception as exc:  # the estimate is reported, never required
        cpu = {"error": f"{type(exc).__name__}: {exc}"}
    return {"workload": "FTLM, J1-J2 L=26 nup=13 J2=0.3 k=0 p=+1 (%d states), %d random vectors, m=%d, "
                        "observables H and sum zz, beta 0.5/1/2" % (n, R, m),
            "batched_samples_per_s": R / t_batch, "sequential_samples_per_s": seq_sample / t_seq,
            "batched_speedup": (R / t_batch) / (seq_sample / t_seq),
            "energy_per_site": [e / L for e in energy],
            "max_rel_diff_batched_vs_sequential": float(np.max(np.abs(
                (acc_b8["H"] - acc_seq["H"]) / acc_seq["H"]))),
            "cpu_port_estimate": cpu}


def section_blocks(qs, torch, L=24, nt=10):
    """evolve on BlockOps: the J1-J2 chain L=24 (J2=0.3) split into its 24
    momentum blocks at nup=12 (2,704,156 states); a seeded random state of
    the nup=12 sector embedded in the 2^24 space, evolved to nt times up to
    t=2 (tol 1e-12, krylov_dim 30): all blocks' recursions on one engine
    against one block at a time (project, evolve, lift)."""
    spec = j1j2_spec(L, 1.0, 0.3)
    terms = [qs.OperatorTerm(o, c) for o, c in spec]
    blocks = [{"kblock": k} for k in range(L)]
    ops = qs.BlockOps(blocks, terms, [], qs.SpinBasis1D, (L,), np.complex128,
                      basis_kwargs={"pauli": False, "nup": L // 2}, compute_all_blocks=True)
    sector = qs.SpinBasis1D(L, nup=L // 2, pauli=False)
    rng = np.random.default_rng(20261203)
    v = rng.standard_normal(sector.Ns) + 1j * rng.standard_normal(sector.Ns)
    psi = qs.project_from(sector, v / np.linalg.norm(v))
    times = np.linspace(0.2, 2.0, nt)
    qs.evolve(ops, psi, 0.0, times[:2])   # warm-up: tiles, graph capture
    torch.cuda.synchronize()
    t = time.perf_counter()
    out = qs.evolve(ops, psi, 0.0, times)
    t_batch = time.perf_counter() - t
    # the same call on device buffers (qs_block_expm with QS_MEM_DEVICE): no
    # 2^L x nt host copy
    from qsgpu import _lib
    hams = list(ops.H_dict.values())
    handles = (ctypes.c_void_p * len(hams))(*[h._h.value for h in hams])
    dpsi = torch.from_numpy(psi).cuda()
    dout = torch.zeros((nt, psi.size), dtype=torch.complex128, device="cuda")
    sc = np.ascontiguousarray(-1j * times)
    torch.cuda.synchronize()
    t = time.perf_counter()
    _lib.check(_lib.load().qs_block_expm(handles, len(hams), 0, ctypes.c_void_p(dpsi.data_ptr()), _lib.ptr(sc), nt,
                                         1e-12, 30, 0, ctypes.c_void_p(dout.data_ptr()), _lib.QS_MEM_DEVICE))
    torch.cuda.synchronize()
    t_dev = time.perf_counter() - t
    dev_err = float(np.max(np.abs(dout.cpu().numpy().T - out)))
    del dout, dpsi
    t = time.perf_counter()
    seq = np.zeros_like(out)
    t_evolve = 0.0
    for h in ops.H_dict.values():
        c = qs.project_to(h.basis, psi)
        t1 = time.perf_counter()
        st = qs.evolve(h, c, 0.0, times)
        t_evolve += time.perf_counter() - t1
        for i in range(nt):
            seq[:, i] += qs.project_from(h.basis, st[:, i])
    t_seq = time.perf_counter() - t
    err = float(np.max(np.linalg.norm(out - seq, axis=0)))
    drift = float(np.max(np.abs(np.linalg.norm(out, axis=0) - 1.0)))
    return {"workload": "BlockOps evolve, J1-J2 L=%d nup=%d J2=0.3, %d momentum blocks (%d states), %d times to "
                        "t=2, tol 1e-12, m=30" % (L, L // 2, len(ops.H_dict), sector.Ns, nt),
            "batched_s": t_batch, "batched_device_buffers_s": t_dev, "device_vs_host_max_diff": dev_err,
            "sequential_s": t_seq, "speedup": t_seq / t_batch,
            "sequential_evolve_only_s": t_evolve, "speedup_device_vs_evolve_only": t_evolve / t_dev,
            "note": "sequential: one block at a time through the public calls (project_to, evolve, project_from "
                    "with host vectors); evolve_only: the per-block evolve calls alone",
            "max_state_diff_batched_vs_sequential": err, "norm_drift": drift}


def section_sweep(qs, torch, sizes=(24, 26, 28, 30), reps=10):
    """Roofline sweep: periodic XXZ (J=1, Delta=0.5, pauli=false) at nup=L/2
    without spatial symmetry, L = 24 .. 30 (N up to 155,117,520; the FP64
    vector alone is 1.24 GB, ten times L2).  Per size: the assembled FP64
    product, the fixed-point form and the matrix-free product on device
    buffers, CUDA events on the operator's stream, a 256 MB buffer written
    between timed products.  Algorithmic bytes of the assembled product:
    4 per stored transition + 26 per row (row length, diagonal, x[r], y[r]);
    the x gathers are extra DRAM traffic once x exceeds L2 (the DRAM bytes
    of the L=28 product are in the profile summary)."""
    import ctypes
    from qsgpu import _lib
    lib = _lib.load()
    peak, _ = load_peaks()
    one, zero = np.array([1.0, 0.0]), np.array([0.0, 0.0])
    stream = torch.cuda.Stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    out = {"workload": "periodic XXZ J=1 Delta=0.5, nup=L/2, no spatial symmetry", "peak_gbs": peak, "sizes": {}}

    def timed(o, xt, yt, flags, n):
        _lib.check(lib.qs_op_set_stream(o._h, ctypes.c_void_p(stream.cuda_stream)))

        def mv():
            _lib.check(lib.qs_op_matvec(o._h, flags, _lib.ptr(one), ctypes.c_void_p(xt.data_ptr()), _lib.QS_F64,
                                        _lib.ptr(zero), ctypes.c_void_p(yt.data_ptr()), _lib.QS_F64, 1,
                                        _lib.QS_MEM_DEVICE))
        for _ in range(3):
            mv()
        torch.cuda.synchronize()
        ts = []
        with torch.cuda.stream(stream):
            for _ in range(n):
                flush.zero_()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                mv()
                e1.record(stream)
                ts.append((e0, e1))
        torch.cuda.synchronize()
        return float(np.mean([a.elapsed_time(b) for a, b in ts]))

    for L in sizes:
        spec = xxz_spec(L)
        terms = [qs.OperatorTerm(o, c) for o, c in spec]
        torch.cuda.synchronize()
        t = time.perf_counter()
        b = qs.SpinBasis1D(L, nup=L // 2, pauli=False)
        t_basis = time.perf_counter() - t
        t = time.perf_counter()
        H = qs.Hamiltonian(b, terms)
        torch.cuda.synchronize()
        t_asm = time.perf_counter() - t
        n, nnz = b.Ns, H.nnz
        x = torch.from_numpy(np.random.default_rng(20261203).standard_normal(n)).cuda()
        y = torch.empty_like(x)
        byts = 4 * nnz + 26 * n
        ms64 = timed(H, x, y, 0, reps)
        y64 = y.clone()
        msfx = timed(H, x, y, _lib.QS_FIXED_POINT, reps)
        fx_err = float((y - y64).norm() / y64.norm())
        del H
        op = qs.QuantumLinearOperator(b, terms)
        msmf = timed(op, x, y, 0, 3)
        mf_err = float((y - y64).norm() / y64.norm())
        del op, x, y, y64
        torch.cuda.empty_cache()
        out["sizes"][str(L)] = {
            "N": n, "nnz": nnz, "basis_s": round(t_basis, 3), "assemble_s": round(t_asm, 3),
            "bytes_per_product": byts,
            "fp64_ms": ms64, "fp64_gbs": byts / ms64 / 1e6, "fp64_frac": byts / ms64 / 1e6 / peak,
            "fixed_point_ms": msfx, "fixed_point_gbs": byts / msfx / 1e6, "fixed_point_frac": byts / msfx / 1e6 / peak,
            "fixed_point_rel_err": fx_err,
            "matrix_free_ms": msmf, "matrix_free_rel_diff": mf_err}
    del flush
    # CPU baseline: the oracle's restatement of the reference's own algorithm
    # (serial scatter with a lookup per generated state, 1 thread), one product
    # of the smallest sweep size
    try:
        import oracle
        L = sizes[0]
        spec = xxz_spec(L)
        ref = oracle.RefBasis(L, nup=L // 2, pauli=False)
        ct = oracle.consolidate_terms(spec)
        d = ref.extract_diagonal(ct)
        pk = oracle.pack_terms(ct)
        xh = np.random.default_rng(20261203).standard_normal(len(d))
        t = time.perf_counter()
        ref.qlo_matvec(ct, xh, total_diag=d, packed=pk)
        cpu_ms = (time.perf_counter() - t) * 1e3
        gpu = out["sizes"][str(L)]
        out["cpu_reference_algorithm"] = {"L": L, "ms_per_product": cpu_ms, "cores": 1,
                                          "vs_fp64_assembled": cpu_ms / gpu["fp64_ms"],
                                          "vs_matrix_free": cpu_ms / gpu["matrix_free_ms"]}
    except Exception as exc:  # the baseline must not hide the GPU figures
        out["cpu_reference_algorithm"] = {"error": f"{type(exc).__name__}: {exc}"}
    return out


def torus_blocks(Lx, Ly):
    """Site maps of the Lx x Ly torus (site = x + Lx y, zero-based): the two
    translations, the x reflection and the spin flip (negative entries)."""
    site = lambda x, y: (x % Lx) + Lx * (y % Ly)  # noqa: E731
    sites = [(x, y) for y in range(Ly) for x in range(Lx)]
    return ([site(x + 1, y) for x, y in sites], [site(x, y + 1) for x, y in sites],
            [site(Lx - 1 - x, y) for x, y in sites], [-(i + 1) for i in range(Lx * Ly)])


def section_general(qs, torch, Lx=6, Ly=5, J2=0.5):
    """SpinBasisGeneral on a 2D lattice: the J1-J2 square lattice on the
    Lx x Ly torus at half filling, sector k = (0, 0), x reflection even, spin
    flip even; basis build, assembly and the Lanczos ground state (k = 1,
    tol 1e-10) in FP64 and double-float.  The bench runs the 6 x 6
    Heisenberg torus (L = 36, 9,075,135,300 parent states)."""
    L = Lx * Ly
    Tx, Ty, Px, Z = torus_blocks(Lx, Ly)
    site = lambda x, y: (x % Lx) + Lx * (y % Ly) + 1  # noqa: E731
    bonds = []
    for y in range(Ly):
        for x in range(Lx):
            bonds += [(1.0, site(x, y), site(x + 1, y)), (1.0, site(x, y), site(x, y + 1)),
                      (J2, site(x, y), site(x + 1, y + 1)), (J2, site(x, y), site(x + 1, y - 1))]
    terms = [qs.OperatorTerm("+-", [(j / 2, a, b) for j, a, b in bonds]),
             qs.OperatorTerm("-+", [(j / 2, a, b) for j, a, b in bonds]),
             qs.OperatorTerm("zz", [(j, a, b) for j, a, b in bonds])]
    torch.cuda.synchronize()
    t = time.perf_counter()
    b = qs.SpinBasisGeneral(L, nup=L // 2, pauli=False, Tx=(Tx, 0), Ty=(Ty, 0), Px=(Px, 0), Z=(Z, 0))
    t_basis = time.perf_counter() - t
    t = time.perf_counter()
    H = qs.Hamiltonian(b, terms)
    t_asm = time.perf_counter() - t
    model = "Heisenberg model" if J2 == 0 else "J1-J2 square lattice (J2=%.2g)" % J2
    out = {"workload": "%s on the %dx%d torus, nup=%d, k=(0,0), Px=+1, Z=+1: %d states, nnz=%d" % (
        model, Lx, Ly, L // 2, b.Ns, H.nnz),
           "basis_build_s": t_basis, "assemble_s": t_asm, "group_order": b.group_order}
    for prec in ("fp64", "fp64df"):
        qs.eigsh(H, k=1, which="SA", tol=1e-10, return_eigenvectors=False, precision=prec)
        torch.cuda.synchronize()
        t = time.perf_counter()
        e0 = qs.eigsh(H, k=1, which="SA", tol=1e-10, return_eigenvectors=False, precision=prec)[0]
        out["lanczos_s_" + prec] = time.perf_counter() - t
        out["e0_per_site_" + prec] = float(e0) / L
    return out


def serving_requests(n_req, rate, seed=20261203):
    """The served mix: Poisson arrivals, L uniform in {18, 20, ..., 30}, nup
    uniform in [L/2-2, L/2], kblock uniform in [0, L), 70 % eigsh k=1 (tol
    1e-10) and 30 % evolve to t ~ U[0.5, 5] (krylov_dim 30, tol 1e-9) on the
    J1-J2 chain (J2 = 0.5), seeded start vectors."""
    rng = np.random.default_rng(seed)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, n_req))
    reqs = []
    for i in range(n_req):
        L = int(rng.choice(np.arange(18, 31, 2)))
        nup = int(rng.integers(L // 2 - 2, L // 2 + 1))
        k = int(rng.integers(0, L))
        kind = "eigsh" if rng.random() < 0.7 else "evolve"
        t = float(rng.uniform(0.5, 5.0))
        reqs.append({"arrival": float(arrivals[i]), "L": L, "nup": nup, "kblock": k, "kind": kind, "t": t,
                     "seed": 1000 + i})
    return reqs


def section_c5(qs, torch, n_req=2000, rate=200.0, budget_gb=150.0, stride=10):
    """Config 5: the request loop under Poisson arrivals; p50/p99 latency
    (completion - arrival) and solves/s of the served forms (FP64, double-
    float, FP32 eigsh + FP64 polish), against the plain FP64 path: one request
    at a time on a stratified sample (every `stride`-th request), (i) with
    each sample operator built beforehand (solve time only, the same operator
    reuse a server cache would give at best) and (ii) building each request's
    operator as it arrives."""
    import threading
    reqs = serving_requests(n_req, rate)
    terms = {}

    def terms_for(L):
        if L not in terms:
            terms[L] = [qs.OperatorTerm(o, c) for o, c in j1j2_spec(L, 1.0, 0.5)]
        return terms[L]

    def basis_of(r):
        return dict(L=r["L"], nup=r["nup"], pauli=False, kblock=r["kblock"])

    def solve(H, r):
        if r["kind"] == "eigsh":
            qs.eigsh(H, k=1, which="SA", tol=1e-10, return_eigenvectors=False)
        else:
            rng = np.random.default_rng(r["seed"])
            v = rng.standard_normal(H.Ns) + 1j * rng.standard_normal(H.Ns)
            qs.evolve(H, v / np.linalg.norm(v), 0.0, [r["t"]], tol=1e-9, krylov_dim=30)

    sample = reqs[::stride]
    # (ii) builds included
    torch.cuda.synchronize()
    t = time.perf_counter()
    for r in sample:
        H = qs.Hamiltonian(qs.SpinBasis1D(**basis_of(r)), terms_for(r["L"]))
        solve(H, r)
        del H
    t_build = time.perf_counter() - t
    # (i) operators built beforehand, one per distinct sector of the sample
    ops = {}
    for r in sample:
        key = (r["L"], r["nup"], r["kblock"])
        if key not in ops:
            ops[key] = qs.Hamiltonian(qs.SpinBasis1D(**basis_of(r)), terms_for(r["L"]))
    torch.cuda.synchronize()
    t = time.perf_counter()
    for r in sample:
        solve(ops[(r["L"], r["nup"], r["kblock"])], r)
    t_pre = time.perf_counter() - t
    del ops
    seq_rate = len(sample) / t_pre
    out = {"workload": "%d requests, Poisson %.0f/s, L in 18..30 (even), J1-J2 J2=0.5, 70%% eigsh k=1 tol 1e-10, "
                       "30%% evolve t~U[0.5,5] m=30 tol 1e-9, HBM budget %.0f GB" % (n_req, rate, budget_gb),
           "sequential_fp64_sample": f"every {stride}th request ({len(sample)} requests)",
           "sequential_fp64_prebuilt_solves_per_s": seq_rate,
           "sequential_fp64_with_builds_solves_per_s": len(sample) / t_build,
           "speedup_baseline": "sequential_fp64_prebuilt_solves_per_s (operators built outside the timed loop)"}
    served = {}
    for name, prec, policy in (("fp64", "fp64", "fifo"), ("fp64df", "fp64df", "fifo"),
                               ("fp64df_smallest_first", "fp64df", "sjf"), ("fp32_smallest_first", "fp32", "sjf")):
        srv = qs.Server(hbm_budget_gb=budget_gb, precision=prec, policy=policy)
        tickets = [None] * n_req
        t0 = time.perf_counter()

        def client():
            for i, r in enumerate(reqs):
                dt = r["arrival"] - (time.perf_counter() - t0)
                if dt > 0:
                    time.sleep(dt)
                if r["kind"] == "eigsh":
                    tickets[i] = srv.submit_eigsh(basis_of(r), terms_for(r["L"]), k=1, tol=1e-10, seed=r["seed"])
                else:
                    tickets[i] = srv.submit_evolve(basis_of(r), terms_for(r["L"]), r["t"], tol=1e-9, krylov_dim=30,
                                                   seed=r["seed"], want_vector=False)
        th = threading.Thread(target=client)
        th.start()
        th.join()
        res = [srv.wait(tk, timeout=3600) for tk in tickets]
        wall = time.perf_counter() - t0
        lat = np.array([x["done_s"] - x["submit_s"] for x in res])
        first = min(x["submit_s"] for x in res)
        last = max(x["done_s"] for x in res)
        st = srv.stats()
        srv.close()
        served[name] = n_req / (last - first)
        out[name] = {"policy": policy, "solves_per_s": served[name], "wall_s": wall,
                     "p50_latency_ms": float(np.percentile(lat, 50) * 1e3),
                     "p99_latency_ms": float(np.percentile(lat, 99) * 1e3),
                     "mean_latency_ms": float(lat.mean() * 1e3),
                     "operator_builds": st["builds"], "cache_hits": st["cache_hits"],
                     "peak_device_gb": st["peak_bytes"] / 1e9, "failed": st["failed"],
                     "speedup_vs_sequential_fp64": served[name] / seq_rate}
    out["served_fp64_continuous_batching_speedup"] = served["fp64"] / seq_rate
    out["offered_load_note"] = (
        "arrivals (%.0f/s) exceed every served throughput (%.1f-%.1f solves/s), so the queue grows for the whole "
        "run and the latencies are dominated by queueing" % (rate, min(served.values()), max(served.values())))
    return out


def profile_range(kind):
    """One unit of work inside cudaProfilerStart/Stop, after warm-up, for
    `ncu --profile-from-start off`: a product of the default sector in FP64,
    FP32, double-float or fixed point ("product64", "product32", "productdf",
    "productfx"), its
    matrix-free product ("matrixfree"), one Lanczos ground state of it
    ("lanczos64", "lanczosdf"), one batched double-float ground-state solve
    of all J1-J2 sectors at L = 20, 24 or 26 ("batch20", "batch24",
    "batch26"; "batch20_fp64", "batch26_fp64" in FP64; the L = 20 sectors run
    on the cluster step), or the 32 batched m = 100 Lanczos recurrences of
    the FTLM workload ("ftlm")."""
    import torch
    import qsgpu as qs
    if kind == "ftlm":
        L = 26
        b = qs.SpinBasis1D(L, nup=13, pauli=False, kblock=0, pblock=1)
        H = qs.Hamiltonian(b, [qs.OperatorTerm(o, c) for o, c in j1j2_spec(L, 1.0, 0.3)])
        V0 = np.random.default_rng(20261203).standard_normal((32, b.Ns)).T
        qs.lanczos_batch(H, V0[:, :2], 100)
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        t = time.perf_counter()
        out = qs.lanczos_batch(H, V0, 100)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_range": kind, "N": b.Ns, "E0": float(out[0][0][0]), "seconds": dt}))
        return
    if kind in ("lanczos64", "lanczosdf"):
        L = 32
        b = qs.SpinBasis1D(L, nup=16, pauli=False, kblock=0, pblock=1, zblock=1)
        H = qs.Hamiltonian(b, [qs.OperatorTerm(o, c) for o, c in j1j2_spec(L, 1.0, 0.5)])
        prec = "fp64" if kind == "lanczos64" else "fp64df"
        qs.eigsh(H, k=1, which="SA", tol=1e-10, return_eigenvectors=False, precision=prec)
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        t = time.perf_counter()
        v = qs.eigsh(H, k=1, which="SA", tol=1e-10, return_eigenvectors=False, precision=prec)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_range": kind, "e0": float(v[0]), "seconds": dt}))
        return
    if kind == "sweep28":
        # one assembled FP64 product of the XXZ L=28 sector without spatial
        # symmetry (N = 40,116,600; x 321 MB, the packed words 2.3 GB)
        import ctypes
        from qsgpu import _lib
        lib = _lib.load()
        L = 28
        b = qs.SpinBasis1D(L, nup=L // 2, pauli=False)
        H = qs.Hamiltonian(b, [qs.OperatorTerm(o, c) for o, c in xxz_spec(L)])
        one, zero = np.array([1.0, 0.0]), np.array([0.0, 0.0])
        xt = torch.from_numpy(np.random.default_rng(20261203).standard_normal(b.Ns)).cuda()
        yt = torch.empty_like(xt)

        def mv():
            _lib.check(lib.qs_op_matvec(H._h, 0, _lib.ptr(one), ctypes.c_void_p(xt.data_ptr()), _lib.QS_F64,
                                        _lib.ptr(zero), ctypes.c_void_p(yt.data_ptr()), _lib.QS_F64, 1,
                                        _lib.QS_MEM_DEVICE))
        for _ in range(3):
            mv()
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        mv()
        torch.cuda.synchronize()
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_range": kind, "N": b.Ns, "nnz": H.nnz, "ynorm": float(yt.norm())}))
        return
    if kind.startswith("product") or kind == "matrixfree":
        L = 32
        b = qs.SpinBasis1D(L, nup=16, pauli=False, kblock=0, pblock=1, zblock=1)
        terms = [qs.OperatorTerm(o, c) for o, c in j1j2_spec(L, 1.0, 0.5)]
        if kind == "matrixfree":
            H = qs.QuantumLinearOperator(b, terms)
        else:
            H = qs.Hamiltonian(b, terms)
        prec = {"product64": "fp64", "product32": "fp32", "productdf": "fp64df", "productfx": "fp64fx",
                "matrixfree": "fp64"}[kind]
        x = np.random.default_rng(20261203).standard_normal(b.Ns)
        # device buffers (what the bench times): one launch is one full-range
        # product
        import ctypes
        from qsgpu import _lib
        lib = _lib.load()
        one, zero = np.array([1.0, 0.0]), np.array([0.0, 0.0])
        code = _lib.QS_F32 if prec == "fp32" else _lib.QS_F64
        xt = torch.from_numpy(x.astype(np.float32) if prec == "fp32" else x).cuda()
        yt = torch.empty_like(xt)
        flags = {"fp64df": _lib.QS_DOUBLE_FLOAT, "fp64fx": _lib.QS_FIXED_POINT}.get(prec, 0)

        def mv():
            _lib.check(lib.qs_op_matvec(H._h, flags, _lib.ptr(one), ctypes.c_void_p(xt.data_ptr()), code,
                                        _lib.ptr(zero), ctypes.c_void_p(yt.data_ptr()), code, 1, _lib.QS_MEM_DEVICE))
        for _ in range(3):
            mv()
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        mv()
        torch.cuda.synchronize()
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_range": kind, "N": b.Ns, "ynorm": float(yt.double().norm())}))
        return
    spec = kind[len("batch"):].split("_")
    L = int(spec[0])
    prec = spec[1] if len(spec) > 1 else "fp64df"
    terms = [qs.OperatorTerm(o, c) for o, c in j1j2_spec(L, 1.0, 0.3)]
    syms = []
    for k in range(L):
        syms += [dict(kblock=k, pblock=1), dict(kblock=k, pblock=-1)] if k in (0, L // 2) else [dict(kblock=k)]
    ops = [qs.Hamiltonian(qs.SpinBasis1D(L, nup=L // 2, pauli=False, **sy), terms) for sy in syms]
    qs.eigsh_batch(ops, k=1, tol=1e-10, precision=prec)
    torch.cuda.synchronize()
    torch.cuda.profiler.start()
    t = time.perf_counter()
    qs.eigsh_batch(ops, k=1, tol=1e-10, precision=prec)
    torch.cuda.synchronize()
    dt = time.perf_counter() - t
    torch.cuda.profiler.stop()
    print(json.dumps({"profile_range": kind, "sectors": len(ops), "states": sum(o.Ns for o in ops), "seconds": dt}))


def run_ours(args, wl, world, rank, local):
    import torch
    torch.cuda.set_device(local)
    import qsgpu as qs
    from qsgpu import _lib
    from qsgpu import build as qbuild
    qbuild.build()
    lib = _lib.load()
    dev = torch.device("cuda", local)
    L, nup = wl["L"], wl["nup"]
    spec = j1j2_spec(L, 1.0, wl["J2"])
    terms = [qs.OperatorTerm(o, c) for o, c in spec]
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    basis = qs.SpinBasis1D(L, nup=nup, pauli=False, **wl["sym"])
    t_basis = time.perf_counter() - t0
    t0 = time.perf_counter()
    H = qs.Hamiltonian(basis, terms)          # assembled on the device (the reference's H.data)
    t_asm = time.perf_counter() - t0
    op = qs.QuantumLinearOperator(basis, terms)  # matrix-free
    n = basis.Ns
    nnz = H.nnz
    # a dedicated stream: the engine launches on it and the CUDA events below
    # are recorded on it
    stream = torch.cuda.Stream(dev)
    torch.cuda.set_stream(stream)
    for o in (H, op):
        _lib.check(lib.qs_op_set_stream(o._h, ctypes.c_void_p(stream.cuda_stream)))
    g = torch.Generator(device="cpu").manual_seed(20261203 + rank)
    xh = torch.randn(n, generator=g, dtype=torch.float64)
    x = xh.to(dev)
    y = torch.empty_like(x)
    x32 = x.float()
    y32 = torch.empty_like(x32)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)  # 256 MB > L2
    one = np.array([1.0, 0.0])
    zero = np.array([0.0, 0.0])

    def mv(o, xt, yt, code, flags=0):
        _lib.check(lib.qs_op_matvec(o._h, flags, _lib.ptr(one), ctypes.c_void_p(xt.data_ptr()), code, _lib.ptr(zero),
                                    ctypes.c_void_p(yt.data_ptr()), code, 1, _lib.QS_MEM_DEVICE))

    def timed(o, xt, yt, code, steps, warmup, flags=0):
        for _ in range(warmup):
            mv(o, xt, yt, code, flags)
        torch.cuda.synchronize()
        barrier(world)
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        l0 = lib.qs_launch_count()
        for s, e in ev:
            flush.zero_()
            s.record(stream)
            mv(o, xt, yt, code, flags)
            e.record(stream)
        torch.cuda.synchronize()
        launches = lib.qs_launch_count() - l0
        return [s.elapsed_time(e) for s, e in ev], launches

    # algorithmic (compulsory) HBM bytes of one product: 4 per stored
    # transition, a 2-byte row length, the 2-byte stabiliser code, the
    # diagonal, x[r] and y[r]
    asm_bytes64 = 4 * nnz + n * (2 + 2 + 3 * 8)
    asm_bytes32 = 4 * nnz + n * (2 + 2 + 3 * 4)
    mf_bytes64 = n * (4 + 2 + 8 + 8 + 8)
    clocks = ClockSampler()
    clocks.start()
    ms64, launches = timed(H, x, y, _lib.QS_F64, args.steps, args.warmup)
    y_native = y.clone()
    ydf = torch.empty_like(x)
    msdf, _ = timed(H, x, ydf, _lib.QS_F64, args.steps, args.warmup, _lib.QS_DOUBLE_FLOAT)
    df_err = float((ydf - y_native).norm() / y_native.norm())
    # fixed-point row sums (FP64 vectors, integer sums per amplitude class)
    yfx = torch.empty_like(x)
    msfx, _ = timed(H, x, yfx, _lib.QS_F64, args.steps, args.warmup, _lib.QS_FIXED_POINT)
    fx_err = float((yfx - y_native).norm() / y_native.norm())
    fx_maxerr = float((yfx - y_native).abs().max() / y_native.abs().max())
    ms32, _ = timed(H, x32, y32, _lib.QS_F32, args.steps, args.warmup)
    mf_steps = max(3, min(args.steps, 10))
    ms_mf, _ = timed(op, x, y, _lib.QS_F64, mf_steps, 2)
    # e2e through the C ABI with host buffers (pinned), copies inside the step
    xp = torch.empty(n, dtype=torch.float64, pin_memory=True)
    xp.copy_(xh)
    yp = torch.empty(n, dtype=torch.float64, pin_memory=True)
    e2e_t = []
    for it in range(args.warmup + args.steps):
        torch.cuda.synchronize()
        t = time.perf_counter()
        _lib.check(lib.qs_op_matvec(H._h, 0, _lib.ptr(one), ctypes.c_void_p(xp.data_ptr()), _lib.QS_F64,
                                    _lib.ptr(zero), ctypes.c_void_p(yp.data_ptr()), _lib.QS_F64, 1,
                                    _lib.QS_MEM_HOST))
        if it >= args.warmup:
            e2e_t.append(time.perf_counter() - t)
    # several right-hand sides (mul!(Y, H, X), X n x 8 on the device): one pass
    # over the words for the 8 columns against 8 single products
    R = 8
    XR = torch.randn(R, n, generator=g, dtype=torch.float64).to(dev)
    YR = torch.empty_like(XR)

    def mv_many(xt, yt, code, nrhs):
        _lib.check(lib.qs_op_matvec(H._h, 0, _lib.ptr(one), ctypes.c_void_p(xt.data_ptr()), code, _lib.ptr(zero),
                                    ctypes.c_void_p(yt.data_ptr()), code, nrhs, _lib.QS_MEM_DEVICE))

    def time_many(xt, yt, code, reps=5):
        for _ in range(2):
            mv_many(xt, yt, code, R)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        tot = 0.0
        for _ in range(reps):
            flush.zero_()
            e0.record(stream)
            mv_many(xt, yt, code, R)
            e1.record(stream)
            torch.cuda.synchronize()
            tot += e0.elapsed_time(e1)
        return tot / reps
    mm64 = time_many(XR, YR, _lib.QS_F64)
    XR32, YR32 = XR.float(), torch.empty_like(XR.float())
    mm32 = time_many(XR32, YR32, _lib.QS_F32)
    multi_rhs = {"columns": R, "fp64_ms": mm64, "fp64_vs_one_product": mm64 / float(np.mean(ms64)),
                 "fp64_column_loop_ms": R * float(np.mean(ms64)),
                 "fp32_ms": mm32, "fp32_vs_one_product": mm32 / float(np.mean(ms32)),
                 "fp32_column_loop_ms": R * float(np.mean(ms32)),
                 "note": "device buffers, one pass over the sliced-ELL words per 8 columns; the FP64 form stays "
                         "bound by one FP64 multiply-add per nonzero and column"}
    del XR, YR, XR32, YR32
    # Lanczos ground state on the assembled operator: FP64, FP32 + FP64 polish and
    # double-float; one warm-up solve each (tile tuning, graph capture), then the
    # mean of three
    solves = {}
    for prec in ("fp64", "fp32", "fp64df"):
        qs.eigsh(H, k=1, which="SA", tol=1e-10, v0=xh.numpy(), return_eigenvectors=False, precision=prec)
        dts = []
        for _ in range(3):
            info = {}
            torch.cuda.synchronize()
            t = time.perf_counter()
            vals = qs.eigsh(H, k=1, which="SA", tol=1e-10, v0=xh.numpy(), return_eigenvectors=False,
                            precision=prec, info=info)
            dts.append(time.perf_counter() - t)
        solves[prec] = dict(seconds=float(np.mean(dts)), e0=float(vals[0]), matvecs=info.get("matvecs"),
                            restarts=info.get("restarts"))
    clk = clocks.stop()

    # the FP64 roofline: one FP64 multiply-add per stored nonzero, plus the
    # diagonal term and the row scale per row, against this GPU's measured FP64
    # FMA throughput
    fma_rate = ctypes.c_double(0.0)
    _lib.check(lib.qs_fp64_fma_rate(ctypes.byref(fma_rate)))
    fma_per_step = nnz + 2 * n
    t_step = max_over_ranks(world, float(np.mean(ms64)) / 1e3, dev)
    value = replica_value(world, asm_bytes64, t_step)
    peak, peak_kind = load_peaks()
    achieved = asm_bytes64 / (float(np.mean(ms64)) / 1e3) / 1e9
    e2e_mean = max_over_ranks(world, float(np.mean(e2e_t)), dev)
    e2e_val = replica_value(world, asm_bytes64, e2e_mean)
    rel_e0 = abs(solves["fp32"]["e0"] - solves["fp64"]["e0"]) / abs(solves["fp64"]["e0"])
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            import oracle
            oracle.lib()
            nthreads = os.cpu_count() or 1
            spr, rows, _, _, tt = cpu_port_sample(wl, nthreads, target_s=10.0)
            cpu = {"value": asm_bytes64 / n / spr / 1e9, "unit": "GB/s", "cores": nthreads, "kind": "port",
                   "sample": f"{rows} contiguous rows of {n} ({tt:.1f} s of matvec), representative-space "
                             "restatement of the reference matvec on all host cores"}
        except Exception as exc:  # the baseline is reported, never required
            cpu = {"value": None, "unit": "GB/s", "cores": os.cpu_count(), "kind": "port",
                   "sample": f"failed: {exc}"}
    sections = {}
    if rank == 0 and not args.no_sections:
        def timed_events(o, xh_np, reps):
            xt = torch.from_numpy(np.ascontiguousarray(xh_np)).to(dev)
            yt = torch.empty_like(xt)
            _lib.check(lib.qs_op_set_stream(o._h, ctypes.c_void_p(stream.cuda_stream)))
            for _ in range(5):
                mv(o, xt, yt, _lib.QS_F64)
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(reps):
                mv(o, xt, yt, _lib.QS_F64)
            e1.record(stream)
            torch.cuda.synchronize()
            return e0.elapsed_time(e1) / reps
        for name, fn in (("c1_xxz_L16", lambda: section_c1(qs, torch, timed_events)),
                         ("c4_batched_sectors_L26", lambda: section_c4(qs, torch)),
                         ("c3_tfim_L30_evolve", lambda: section_c3(qs, torch)),
                         ("ftlm_L26", lambda: section_ftlm(qs, torch)),
                         ("blocks_L24_evolve", lambda: section_blocks(qs, torch)),
                         ("general_6x6_heisenberg", lambda: section_general(qs, torch, Lx=6, Ly=6, J2=0.0)),
                         ("roofline_sweep_xxz", lambda: section_sweep(qs, torch)),
                         ("c5_serving", lambda: section_c5(qs, torch, n_req=args.serve_requests))):
            if args.only_section and name != args.only_section:
                continue
            try:
                sections[name] = fn()
            except Exception as exc:  # a failing side workload must not hide the headline
                sections[name] = {"error": f"{type(exc).__name__}: {exc}"}
    if rank != 0:
        return
    line = {
        "metric": METRIC, "value": value, "unit": "GB/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": t_step * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": wl["desc"], "N": n, "nnz": nnz,
                   "step": "one H.v of the assembled Hamiltonian over the sector, x/y resident in HBM",
                   "bytes_per_step": asm_bytes64, "l2": "256 MB buffer written between timed steps",
                   "basis_build_s": round(t_basis, 3), "assemble_s": round(t_asm, 3),
                   "parallelism": f"replicas x{world}"},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                     "traffic": wl.get("traffic"), "traffic_source": wl.get("traffic_source"),
                     "peak_kind": peak_kind,
                     "kernel": "sell_kernel (assembled H.v, sliced ELL)"},
        "fp64_roofline": {"bound": "fp64 pipe", "achieved": fma_per_step / (float(np.mean(ms64)) / 1e3) / 1e12,
                          "peak": fma_rate.value / 1e12, "unit": "T FMA/s",
                          "frac": fma_per_step / (float(np.mean(ms64)) / 1e3) / fma_rate.value,
                          "fma_per_step": fma_per_step,
                          "peak_kind": "measured in this run (qs_fp64_fma_rate: chained FP64 FMA kernel)"},
        "e2e": {"value": e2e_val, "unit": "GB/s", "h2d_bytes_per_step": n * 8, "d2h_bytes_per_step": n * 8},
        "gpu_launches": int(launches),
        "clocks": clk,
        "fp32_form": {"value": asm_bytes32 / (float(np.mean(ms32)) / 1e3) / 1e9, "unit": "GB/s",
                      "ms_per_step": float(np.mean(ms32)),
                      "speedup_vs_fp64": float(np.mean(ms64)) / float(np.mean(ms32))},
        "fp64_double_float_form": {"value": asm_bytes64 / (float(np.mean(msdf)) / 1e3) / 1e9, "unit": "GB/s",
                                   "ms_per_step": float(np.mean(msdf)),
                                   "frac_of_peak": asm_bytes64 / (float(np.mean(msdf)) / 1e3) / 1e9 / peak,
                                   "rel_err_vs_native_fp64": df_err,
                                   "speedup_vs_fp64": float(np.mean(ms64)) / float(np.mean(msdf))},
        "fp64_fixed_point_form": {"value": asm_bytes64 / (float(np.mean(msfx)) / 1e3) / 1e9, "unit": "GB/s",
                                  "ms_per_step": float(np.mean(msfx)),
                                  "frac_of_peak": asm_bytes64 / (float(np.mean(msfx)) / 1e3) / 1e9 / peak,
                                  "classes": H.fixed_point_classes,
                                  "rel_err_vs_native_fp64": fx_err, "max_err_rel_to_max_entry": fx_maxerr,
                                  "speedup_vs_fp64": float(np.mean(ms64)) / float(np.mean(msfx)),
                                  "note": "x sqrt(stab) scaled to int64 once per product (two passes over x, "
                                          "included), exact integer row sums, FP64 per row"},
        "matrix_free": {"ms_per_step": float(np.mean(ms_mf)), "unit": "GB/s",
                        "value": mf_bytes64 / (float(np.mean(ms_mf)) / 1e3) / 1e9,
                        "note": "QuantumLinearOperator path: transitions regenerated every product"},
        "lanczos": {"solves_per_s_fp64": 1.0 / solves["fp64"]["seconds"],
                    "solves_per_s_fp32_polished": 1.0 / solves["fp32"]["seconds"],
                    "solves_per_s_fp64_double_float": 1.0 / solves["fp64df"]["seconds"],
                    "fp64df_rel_err": abs(solves["fp64df"]["e0"] - solves["fp64"]["e0"]) / abs(solves["fp64"]["e0"]),
                    "e0": solves["fp64"]["e0"], "fp32_polished_rel_err": rel_e0,
                    "matvecs_fp64": solves["fp64"]["matvecs"], "matvecs_fp32": solves["fp32"]["matvecs"],
                    "tol": 1e-10},
        "latency_ms": {"p50": float(np.percentile(ms64, 50)), "p99": float(np.percentile(ms64, 99))},
        "multi_rhs": multi_rhs,
        "cpu_baseline": cpu,
        "workloads": sections,
    }
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="j1j2_L32_k0_p1_z1", choices=sorted(WORKLOADS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-sections", action="store_true",
                    help="skip the side workloads (XXZ L=16, batched sectors, TFIM evolve, serving)")
    ap.add_argument("--serve-requests", type=int, default=2000, help="requests in the serving workload")
    ap.add_argument("--only-section", default=None, help="run this side workload only (by its JSON key)")
    ap.add_argument("--profile-range", default=None,
                    choices=["product64", "product32", "productdf", "productfx", "sweep28", "matrixfree", "lanczos64", "lanczosdf",
                             "batch20", "batch20_fp64", "batch24", "batch26", "batch26_fp64", "ftlm"],
                    help="run one unit inside cudaProfilerStart/Stop (for ncu --profile-from-start off) and exit")
    args = ap.parse_args()
    if args.profile_range:
        profile_range(args.profile_range)
        return
    if args.warmup < 3:
        args.warmup = 3
    wl = WORKLOADS[args.workload]
    world, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference(args, wl, world, rank)
    else:
        run_ours(args, wl, world, rank, local)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
