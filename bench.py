#!/usr/bin/env python
"""Estimator solves/s on one B200 (or N replicas), mixed vs plain FP64 path.

Workload (default, the 16x16 kicked-Ising solve): open 16x16 square-lattice
PEPS in |0...0>, 20 Floquet steps of RZZ(theta_J = -pi/4) on every edge then
RX(theta_h) on every site (theta_h ~ U[0.2, 1.2] from the seed), chi = 16
(BP at bond dimension 32), BP tolerance 1e-8 / 50 sweeps, sv_min 1e-8;
observable (1/256) sum_i Z_i + 32 random distinct nearest-neighbour Z Z terms
(coefficient 1).  The seed (25, theta_h = 0.3607) is one whose draw lies in
the regime where loopy BP converges on this lattice (see SEED).  Synthetic input: the reference's public inputs are
generated, not loaded.

One step = one full solve (absorb + BP + truncation for every Floquet step,
then the FP64 sum of the Pauli terms).  `value` = solves/s of the mixed
(complex64) path with the problem resident on the device; `e2e` = the same
through the public API from host data (lattice, TPO and terms uploaded,
result read back each solve).  The plain complex128 path is timed on one
solve beside it and |dE| between the two is reported.  Site tensors at
BP time (~3 GB c64, 6 GB c128) exceed the 126 MB L2, so no flush is needed.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (torchrun, one rank per GPU) every rank solves its own replica:
the path does not shard (replicas only); value = N*K solves / max-rank time.
--impl reference times the reference's own algorithm on the host cores
(oracle/_ref/estimator: the unchanged tnbp estimator app on the project's
CPU tensor backend) on a bounded sample of the same workload.
"""
import argparse
import json
import math
import os
import re
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

L_SIDE, CHI, STEPS = 16, 16, 20
THETA_J = -math.pi / 4
BP_TOL, BP_MAXIT, SV_MIN = 1e-8, 50, 1e-8
# theta_h ~ U[0.2, 1.2] from this seed: 0.3607.  The first seed tried
# (20261203, theta_h = 1.038) is outside the regime where loopy BP converges
# on this lattice: from step 7 on its condition never reaches 1e-8 and grows
# after its minimum, so every step runs 50 sweeps and the messages are noise.
SEED = 25
CPU_SAMPLE_STEPS = 5  # Floquet steps of the CPU reference sample
# Served stream: 512 requests, Poisson arrivals 2 ms apart on average, L in
# {4,6,8,10,12}, chi in {8,16,32}, depth in 4..16, theta_h in [0.2,1.2],
# 8-term random observable each.  Its requests at chi 32 on 10x10 and 12x12
# lattices (BP at D = 64; the 11th request is the first) run for ten minutes
# and more each on the plain path, so the default bench serves the first
# SERVED_N requests (a prefix of the same seeded stream; --served-requests
# changes it, --served-only runs that leg alone).
SERVED_SEED, SERVED_TOTAL, SERVED_N = 25, 512, 8
# The escalating server restarts a request in complex128 when one of its BP
# loops runs out of sweeps without its condition ever falling below this.
# Measured on the first 24 requests of the stream (mixed server run twice,
# theta_h and theta_h (1 + 1e-9)): the two requests whose value the
# perturbation moved by more than 1e-6 (1e-1 and 7e-4) had loops whose
# smallest condition was 0.19 and 0.35; every other request's was <= 3.4e-3
# and its value moved by <= 2.4e-7, except one (6x6, chi 32, 13 steps:
# smallest condition 3.1e-3, moved by 1.04e-6) that this threshold leaves on
# the mixed path.
ESC_MIN_COND = 1e-2


METRIC = "estimator solves/s (mixed path; plain FP64 GPU path and |dE| beside)"


def workload_config(theta_h, world):
    return {"workload": f"kicked-Ising {L_SIDE}x{L_SIDE} open PEPS, {STEPS} steps, chi={CHI}, RZZ(-pi/4), RX(theta_h)",
            "theta_h": theta_h, "seed": SEED, "bp_tol": BP_TOL, "bp_max_iter": BP_MAXIT,
            # the mixed path's BP loop stops at max(bp_tol, 1e-7), its rounding
            # floor, or at the first growing condition below 1e-5; the plain
            # path keeps bp_tol
            "bp_tol_effective_mixed": max(BP_TOL, 1e-7),
            "sv_min": SV_MIN, "observable": f"(1/{L_SIDE * L_SIDE}) sum Z_i + 32 NN ZZ",
            "parallelism": f"replicas x{world}",
            "l2": "no flush: site tensors at BP time (~3 GB) exceed the 126 MB L2"}


def workload(seed=SEED):
    rng = np.random.default_rng(seed)
    theta_h = float(rng.uniform(0.2, 1.2))
    n = L_SIDE * L_SIDE
    edges = []
    for iy in range(L_SIDE):
        for ix in range(L_SIDE):
            s = ix + L_SIDE * iy
            if ix + 1 < L_SIDE:
                edges.append((s, s + 1))
            if iy + 1 < L_SIDE:
                edges.append((s, s + L_SIDE))
    zz = rng.choice(len(edges), size=min(32, len(edges)), replace=False)
    lines = [f"{1.0 / n!r} " + "".join("Z" if n - 1 - k == i else "I" for k in range(n)) for i in range(n)]
    for m in sorted(int(x) for x in zz):
        a, b = edges[m]
        lines.append("1.0 " + "".join("Z" if n - 1 - k in (a, b) else "I" for k in range(n)))
    return theta_h, "\n".join(lines) + "\n"


def kicked_ising_qasm(steps, theta_j, theta_h):
    n = L_SIDE * L_SIDE
    out = ["OPENQASM 2.0;", 'include "qelib1.inc";', f"qreg q[{n}];"]
    for _ in range(steps):
        for iy in range(L_SIDE):
            for ix in range(L_SIDE - 1):
                i = ix + L_SIDE * iy
                out.append(f"rzz({theta_j!r}) q[{i}],q[{i + 1}];")
        for iy in range(L_SIDE - 1):
            for ix in range(L_SIDE):
                i = ix + L_SIDE * iy
                out.append(f"rzz({theta_j!r}) q[{i}],q[{i + L_SIDE}];")
        for i in range(n):
            out.append(f"rx({theta_h!r}) q[{i}];")
        out.append("barrier q;")
    return "\n".join(out) + "\n"


def random_observable(rng, n_qubits, n_terms=8):
    """n_terms Pauli strings on 1-4 distinct random qubits, letters uniform in
    {X,Y,Z}, coefficients N(0,1), as `.txt` lines (rightmost char = qubit 0).
    The reference's ClassifyOps keeps 1-qubit and adjacent 2-qubit terms."""
    lines = []
    for _ in range(n_terms):
        k = int(rng.integers(1, 5))
        qs = rng.choice(n_qubits, size=k, replace=False)
        letters = rng.choice(list("XYZ"), size=k)
        chars = ["I"] * n_qubits
        for q, c in zip(qs, letters):
            chars[n_qubits - 1 - int(q)] = str(c)
        lines.append(f"{float(rng.normal())!r} " + "".join(chars))
    return "\n".join(lines) + "\n"


def random_circuit_workload(seed=SEED, L=10, layers=12):
    """Random-circuit estimator: L x L qubits, `layers` layers of U3 (three
    angles uniform in [0, 2pi)) on every qubit followed by CZ on one of four
    edge colourings in cyclic order (horizontal even, horizontal odd,
    vertical even, vertical odd), a barrier after each layer; 64-term random
    observable.  Returns (qasm, pauli text)."""
    rng = np.random.default_rng(seed)
    n = L * L
    out = ["OPENQASM 2.0;", 'include "qelib1.inc";', f"qreg q[{n}];"]
    for layer in range(layers):
        for i in range(n):
            a, b, c = (float(x) for x in rng.uniform(0.0, 2 * math.pi, size=3))
            out.append(f"u3({a!r},{b!r},{c!r}) q[{i}];")
        col = layer % 4
        for iy in range(L):
            for ix in range(L):
                i = ix + L * iy
                if col < 2 and ix % 2 == col and ix + 1 < L:
                    out.append(f"cz q[{i}],q[{i + 1}];")
                if col >= 2 and iy % 2 == col - 2 and iy + 1 < L:
                    out.append(f"cz q[{i}],q[{i + L}];")
        out.append("barrier q;")
    return "\n".join(out) + "\n", random_observable(rng, n, 64)


def estimator_from_qasm(tb, precision, qasm, pauli, chi, clusters=None, per_term=None):
    """QasmToTPO layers, then the estimator loop; returns (sum, terms kept,
    terms dropped).  With a dict `clusters`, every row of the observable is
    also measured (the dropped ones on their tree clusters) into it: the
    all-terms sum and the host time of that measurement.  With a dict
    `per_term`, the kept terms' values are stored in it in the order the
    reference app prints them (one-site terms, then two-site terms, each in
    file order)."""
    edges = tb.EdgesFromQasm(qasm)
    layers = tb.QasmToTPO(qasm, edges)
    terms = tb.load_sparse_pauli(pauli, edges)
    with tb.State(edges, precision) as st:
        for layer in layers:
            tb.AbsorbTPO(st, layer)
            tb.BeliefPropagationLoop(st, BP_TOL, BP_MAXIT)
            tb.Truncation(st, chi, SV_MIN)
        total, per = tb.MeasurePauliSum(st, terms)
        if per_term is not None:
            kinds = np.asarray(terms.kind)
            per_term["one"] = [float(v.real) for v in per[kinds == 1]]
            per_term["two"] = [float(v.real) for v in per[kinds == 2]]
        if clusters is not None:
            t = time.perf_counter()
            all_sum, vals, kinds = tb.MeasurePauliText(st, pauli, clusters=True)
            clusters["ms"] = (time.perf_counter() - t) * 1e3
            clusters["sum"] = all_sum
            clusters["n_cluster_terms"] = int(np.sum(kinds == 3))
            clusters["values"] = vals
    return total, len(terms), terms.dropped


def random_circuit_summary(tb):
    import torch
    qasm, pauli = random_circuit_workload()
    res = {}
    arms = (("mixed", tb.MIXED), ("plain_fp64", tb.C128))
    for _, prec in arms:
        estimator_from_qasm(tb, prec, qasm, pauli, 32)  # warm-up
    # a solve is 15-25 ms of mostly host work: five solves per arm, the arms
    # interleaved, median
    secs = {name: [] for name, _ in arms}
    for _ in range(5):
        for name, prec in arms:
            torch.cuda.synchronize()
            t = time.perf_counter()
            total, kept, dropped = estimator_from_qasm(tb, prec, qasm, pauli, 32)
            torch.cuda.synchronize()
            secs[name].append(time.perf_counter() - t)
            res[name] = {"sum": [total.real, total.imag]}
    for name, _ in arms:
        res[name]["solves_per_s"] = 1.0 / float(np.median(secs[name]))
        res[name]["solve_ms"] = [round(x * 1e3, 2) for x in secs[name]]
    res["speedup"] = res["mixed"]["solves_per_s"] / res["plain_fp64"]["solves_per_s"]
    res["dE"] = abs(complex(*res["mixed"]["sum"]) - complex(*res["plain_fp64"]["sum"]))
    res["terms_kept"], res["terms_dropped"] = kept, dropped
    # the full observable: the dropped terms measured on their tree clusters
    cm, cp = {}, {}
    estimator_from_qasm(tb, tb.MIXED, qasm, pauli, 32, clusters=cm)
    estimator_from_qasm(tb, tb.C128, qasm, pauli, 32, clusters=cp)
    res["all_terms"] = {"sum_mixed": [cm["sum"].real, cm["sum"].imag], "sum_plain_fp64": [cp["sum"].real, cp["sum"].imag],
                        "dE": abs(cm["sum"] - cp["sum"]),
                        "dterm_max": float(np.max(np.abs(cm["values"] - cp["values"]))),
                        "cluster_terms": cm["n_cluster_terms"], "measure_ms_mixed": cm["ms"],
                        "note": "terms the reference drops measured on tree clusters (not in the reference)"}
    res["workload"] = ("random circuit 10x10, 12 layers U3 + CZ (4 colourings, cyclic), chi 32, "
                       "64-term observable (the reference drops >2-qubit and non-adjacent terms); host wall clock")
    # host cost of a served QASM request's TPO (built once per program and
    # cached): QasmToTPO, then OptTPObySVD on every layer, against the mixed
    # solve it feeds
    edges = tb.EdgesFromQasm(qasm)
    t = time.perf_counter()
    layers = tb.QasmToTPO(qasm, edges)
    t_tpo = time.perf_counter() - t
    t = time.perf_counter()
    for layer in layers:
        tb.OptTPObySVD(edges, layer, 1e-8)
    t_opt = time.perf_counter() - t
    res["host_tpo"] = {"qasm_to_tpo_ms": t_tpo * 1e3, "opt_tpo_by_svd_ms": t_opt * 1e3, "layers": len(layers),
                       "fraction_of_mixed_solve": (t_tpo + t_opt) * res["mixed"]["solves_per_s"],
                       "note": "host (one thread); per distinct program, cached by the server"}
    return res


def served_stream(n, seed=SERVED_SEED, total=SERVED_TOTAL):
    """The first n requests of the seeded served stream (all `total` are drawn
    so that every n gives a prefix of the same stream)."""
    rng = np.random.default_rng(seed)
    reqs, t = [], 0.0
    for _ in range(total):
        t += float(rng.exponential(2e-3))
        L = int(rng.choice([4, 6, 8, 10, 12]))
        chi = int(rng.choice([8, 16, 32]))
        depth = int(rng.integers(4, 17))
        th = float(rng.uniform(0.2, 1.2))
        reqs.append({"t": t, "L": L, "chi": chi, "depth": depth, "theta_h": th,
                     "pauli": random_observable(rng, L * L)})
    return reqs[:n]


def run_served(tb, reqs, precision, escalate=False, esc_min_cond=0.0):
    """Continuous batching (tnbp_server_*): requests are submitted at their
    arrival times (host clock) and the server steps while any is in flight.
    Latency = result available - arrival (host wall clock).  A request whose
    footprint exceeds the GPU's HBM is refused at submission (TNBP_ENOMEM):
    its index goes to `rejected` and it has no value.  With `escalate`, the
    server restarts non-converging requests in complex128."""
    srv = tb.Server(precision, 0, 64)
    t0 = time.perf_counter()
    ids, fin, nxt, rejected, info = {}, {}, 0, [], {}
    try:
        if precision != tb.C128:
            srv.set_escalation(escalate)
            srv.set_escalation_threshold(esc_min_cond)
        while len(fin) + len(rejected) < len(reqs):
            now = time.perf_counter() - t0
            while nxt < len(reqs) and reqs[nxt]["t"] <= now:
                r = reqs[nxt]
                terms = tb.load_sparse_pauli(r["pauli"], tb.bond_square_lattice(r["L"], r["L"]))
                try:
                    ids[nxt] = srv.submit_kicked_ising(r["L"], r["chi"], r["depth"], THETA_J, r["theta_h"], terms,
                                                       BP_TOL, BP_MAXIT, SV_MIN)
                except tb.TnbpError as e:
                    if e.code != tb.ENOMEM:
                        raise
                    rejected.append(nxt)
                nxt += 1
            if len(ids) == len(fin):
                if nxt < len(reqs):
                    time.sleep(max(0.0, reqs[nxt]["t"] - now))
                continue
            srv.step()
            now = time.perf_counter() - t0
            for i, rid in ids.items():
                if i not in fin:
                    try:
                        v = srv.result(rid)
                    except tb.TnbpError:
                        v = complex("nan")  # the request failed; the others go on
                    if v is not None:
                        fin[i] = (now, v)
                        info[i] = srv.info(rid)
    finally:
        srv.close()
    kept = sorted(fin)
    lat = [fin[i][0] - reqs[i]["t"] for i in kept]
    span = max(f[0] for f in fin.values()) - reqs[0]["t"]
    return {i: fin[i][1] for i in kept}, lat, span, info, rejected


def run_plain_fifo(tb, reqs, precision, skip=()):
    """The plain per-job path (State / AbsorbTPO / BeliefPropagationLoop /
    Truncation / MeasurePauliSum), one request at a time in arrival order
    (requests in `skip` are left out)."""
    t0 = time.perf_counter()
    vals, lat, conv = {}, [], {}
    for i, r in enumerate(reqs):
        if i in skip:
            continue
        now = time.perf_counter() - t0
        if now < r["t"]:
            time.sleep(r["t"] - now)
        edges = tb.bond_square_lattice(r["L"], r["L"])
        layer = tb.KickedIsingTPO(edges, THETA_J / 2, 0.0, r["theta_h"] / 2, 1.0)
        ok = True
        with tb.State(edges, precision) as st:
            tpo = st.tpo(layer)
            for _ in range(r["depth"]):
                tb.AbsorbTPO(st, tpo)
                _, c = tb.BeliefPropagationLoop(st, BP_TOL, BP_MAXIT)
                ok = ok and c < BP_TOL
                tb.Truncation(st, r["chi"], SV_MIN)
            tot, _ = tb.MeasurePauliSum(st, tb.load_sparse_pauli(r["pauli"], edges))
        vals[i] = tot
        conv[i] = ok
        lat.append(time.perf_counter() - t0 - r["t"])
    span = time.perf_counter() - t0 - reqs[0]["t"]
    return vals, lat, span, conv


def served_summary(tb, n):
    """The first n requests of the served stream three ways: the mixed server
    with escalation (requests whose BP does not converge are re-run in
    complex128, so every value is within 1e-6 of the plain path), the mixed
    server alone, and the plain complex128 path one request at a time."""
    reqs = served_stream(n)
    esc, lat_e, span_e, info_e, rejected = run_served(tb, reqs, tb.MIXED, escalate=True, esc_min_cond=ESC_MIN_COND)
    mix, lat_m, span_m, info_m, _ = run_served(tb, reqs, tb.MIXED, escalate=False)
    plain, lat_p, span_p, conv = run_plain_fifo(tb, reqs, tb.C128, skip=set(rejected))
    kept = sorted(set(plain) & set(esc) & set(mix))
    dE_e = [abs(esc[i] - plain[i]) for i in kept]
    dE_m = [abs(mix[i] - plain[i]) for i in kept]

    def pct(x, q):
        return float(np.percentile(np.asarray(x) * 1e3, q))

    def arm(span, lat, dE):
        return {"solves_per_s": len(kept) / span, "p50_ms": pct(lat, 50), "p99_ms": pct(lat, 99),
                "dE_max": max(dE), "n_dE_over_1e-6": sum(d > 1e-6 for d in dE), "dE_per_request": dE}
    return {
        "sample": f"first {n} of the seeded {SERVED_TOTAL}-request stream (seed {SERVED_SEED}): Poisson arrivals "
                  "mean 2 ms, L in {4..12 even}, chi in {8,16,32}, depth 4-16, theta_h U[0.2,1.2], "
                  "8-term random observable; latencies on the host clock",
        "requests": [[r["L"], r["chi"], r["depth"], round(r["theta_h"], 4)] for r in reqs],
        "rejected_by_footprint": rejected,
        "measured": kept,
        "mixed_escalating": dict(arm(span_e, lat_e, dE_e), escalation_min_cond=ESC_MIN_COND,
                                 escalated=[i for i in kept if info_e[i]["escalated"]]),
        "mixed": dict(arm(span_m, lat_m, dE_m),
                      bp_stats=[[info_m[i]["unconverged_loops"], info_m[i]["worst_min_cond"],
                                 info_m[i]["worst_final_cond"]] for i in kept],
                      bp_stats_columns=["loops at the iteration limit", "largest smallest condition of those loops",
                                        "largest final condition"]),
        "plain_fp64_fifo": {"solves_per_s": len(kept) / span_p, "p50_ms": pct(lat_p, 50),
                            "p99_ms": pct(lat_p, 99)},
        "speedup_escalating": span_p / span_e,
        "speedup_mixed": span_p / span_m,
        "fp64_bp_converged": [conv[i] for i in kept],
        "note": "dE against the plain complex128 path; where BP does not converge the kept messages carry the "
                "rounding of every earlier sweep amplified, so only escalation keeps those requests within 1e-6",
    }


class ClockSampler:
    """nvidia-smi clocks and throttle reasons during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu):
        self.gpu, self.rows, self.p = gpu, [], None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.p = None
        return self

    def _read(self):
        for line in self.p.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.p:
            self.p.terminate()
            try:
                self.p.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.p.kill()

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4) if len(r) > 5 + i and r[5 + i] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def solve(tb, precision, theta_h, pauli_text, events=None):
    """One estimator solve from host data.  Returns (sum, per-solve stats).
    With `events`, a CUDA event is recorded once the state and TPO are on the
    device (the start of the resident-input timing)."""
    import torch
    h2d = d2h = 0
    edges = tb.bond_square_lattice(L_SIDE, L_SIDE)
    layer = tb.KickedIsingTPO(edges, THETA_J / 2, 0.0, theta_h / 2, 1.0)
    st = tb.State(edges, precision)
    tpo = st.tpo(layer)
    terms = tb.load_sparse_pauli(pauli_text, edges)
    h2d += len(edges) * 8 + layer.op_data.nbytes + layer.edge_rank.nbytes + layer.op_offset.nbytes
    h2d += len(terms) * (4 * 3 + 2 + 16)
    if events is not None:
        torch.cuda.synchronize()
        events.append(torch.cuda.Event(enable_timing=True))
        events[-1].record()
    sweeps = 0
    for _ in range(STEPS):
        tb.AbsorbTPO(st, tpo)
        it, _ = tb.BeliefPropagationLoop(st, BP_TOL, BP_MAXIT)
        sweeps += it
        d2h += 8 * (it + 1)
        tb.Truncation(st, CHI, SV_MIN)
        d2h += st.ne * 12
    total, per = tb.MeasurePauliSum(st, terms)
    d2h += 16 + 16 * len(per)
    stats = dict(sweeps=sweeps, totals=st.sweep_totals(), h2d=h2d, d2h=d2h, per=per)
    st.close()
    return total, stats


def config5_summary(tb, chi=16, steps=24, theta_h=0.6):
    """The large single solve at reduced chi: kicked Ising on the 32x32 open
    lattice, RZZ(-pi/4), RX(0.6), 24 steps, BP tolerance 1e-8 (SV_MIN as
    the headline), observable = every single-site Z (1024) plus every
    nearest-neighbour ZZ (1984), coefficient 1.  chi = 64 as stated needs
    BP at bond dimension 128 (about 3.6 TiB of site tensors), so it cannot
    run on one GPU; this runs chi = 16 (BP at 32) with both paths and
    reports the largest chi whose estimated peak footprint fits the GPU."""
    import torch
    L = 32
    edges = tb.bond_square_lattice(L, L)
    n = L * L
    lines = [f"1.0 " + "".join("Z" if n - 1 - k == i else "I" for k in range(n)) for i in range(n)]
    for a, b in edges:
        lines.append("1.0 " + "".join("Z" if n - 1 - k in (a, b) else "I" for k in range(n)))
    pauli = "\n".join(lines) + "\n"
    terms = tb.load_sparse_pauli(pauli, edges)
    layer = tb.KickedIsingTPO(edges, THETA_J / 2, 0.0, theta_h / 2, 1.0)
    res = {}
    for name, prec in (("mixed", tb.MIXED), ("plain_fp64", tb.C128)):
        torch.cuda.synchronize()
        t = time.perf_counter()
        sweeps = 0
        with tb.State(edges, prec) as st:
            tpo = st.tpo(layer)
            for _ in range(steps):
                tb.AbsorbTPO(st, tpo)
                it, _ = tb.BeliefPropagationLoop(st, 1e-8, BP_MAXIT)
                sweeps += it
                tb.Truncation(st, chi, SV_MIN)
            total, per = tb.MeasurePauliSum(st, terms)
            peak = st.device_bytes()
            tot = st.sweep_totals()
        torch.cuda.synchronize()
        res[name] = {"seconds": time.perf_counter() - t, "sum": [total.real, total.imag], "bp_sweeps": sweeps,
                     "sweep_ms": tot[0] / max(1, tot[3]), "device_bytes_end": peak, "per": per}
    pm, pp = res["mixed"].pop("per"), res["plain_fp64"].pop("per")
    res["dE"] = abs(complex(*res["mixed"]["sum"]) - complex(*res["plain_fp64"]["sum"]))
    res["dterm_max"] = float(np.max(np.abs(pm - pp)))
    res["speedup"] = res["plain_fp64"]["seconds"] / res["mixed"]["seconds"]
    free, total_mem = torch.cuda.mem_get_info()
    fits = {}
    for c in (16, 24, 32, 48, 64):
        fp = tb.footprint_estimate(edges, [2 * c] * len(edges), tb.MIXED)
        fits[c] = {"footprint_gb": fp / 1e9, "fits": fp <= total_mem}
    res["largest_chi_fitting"] = max([c for c, v in fits.items() if v["fits"]], default=None)
    res["footprint_by_chi"] = fits
    res["workload"] = (f"kicked-Ising 32x32, {steps} steps, theta_J=-pi/4, theta_h={theta_h}, chi={chi} "
                       "(stated chi 64 does not fit one GPU), 1024 Z + 1984 ZZ terms; host wall clock per solve")
    # the first BP loop of a shape class runs the wave-budget autotuner
    # inside the solve unless TNBP_AUTOTUNE=0 (one wave, its usual choice)
    res["autotuner_in_solve"] = os.environ.get("TNBP_AUTOTUNE", "1") != "0"
    return res


def max_over_ranks(dist, values, device):
    """Element-wise maximum of per-rank timings (every rank gets it)."""
    import torch
    t = torch.tensor(values, device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t]


def replica_value(world, steps, ms_max):
    """Whole-job solves/s of `world` independent replicas that each ran
    `steps` solves, timed by the slowest rank (weak scaling)."""
    return world * steps / (ms_max / 1e3)


def run_ours(args, rank, world, local_rank):
    import torch
    import tnbp_b200 as tb

    if not torch.cuda.is_available() or not tb.device_available():
        raise SystemExit("bench needs a CUDA device")
    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600), device_id=torch.device("cuda", local_rank))
    theta_h, pauli_text = workload()
    edges = tb.bond_square_lattice(L_SIDE, L_SIDE)

    # warm-up (untimed): same work as a timed step
    for _ in range(args.warmup):
        solve(tb, tb.MIXED, theta_h, pauli_text)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    launches0 = tb.kernel_launches()
    ev_e2e0, ev_res, ev_end = [], [], []
    sums, stats = [], []
    with ClockSampler(local_rank) as clk:
        t_wall = time.perf_counter()
        for _ in range(args.steps):
            torch.cuda.synchronize()
            e0 = torch.cuda.Event(enable_timing=True)
            e0.record()
            ev_e2e0.append(e0)
            s, stt = solve(tb, tb.MIXED, theta_h, pauli_text, events=ev_res)
            torch.cuda.synchronize()
            e1 = torch.cuda.Event(enable_timing=True)
            e1.record()
            ev_end.append(e1)
            sums.append(s)
            stats.append(stt)
        torch.cuda.synchronize()
        t_wall = time.perf_counter() - t_wall
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    launches = tb.kernel_launches() - launches0
    e2e_ms = sum(a.elapsed_time(b) for a, b in zip(ev_e2e0, ev_end))
    res_ms = sum(a.elapsed_time(b) for a, b in zip(ev_res, ev_end))
    if dist:
        e2e_ms, res_ms = max_over_ranks(dist, [e2e_ms, res_ms], "cuda")
    if rank != 0:
        dist.destroy_process_group()
        return
    K = args.steps
    value = replica_value(world, K, res_ms)
    e2e_value = replica_value(world, K, e2e_ms)
    tot_ms = sum(s["totals"][0] for s in stats)
    tot_fl = sum(s["totals"][1] for s in stats)
    tot_by = sum(s["totals"][2] for s in stats)
    n_sw = sum(s["totals"][3] for s in stats)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except (OSError, ValueError):
        pass
    tf_peak = peaks.get("bf16_tflops_sustained") or 1400.0
    achieved = (tot_fl / n_sw) / ((tot_ms / n_sw) / 1e3) / 1e12 if n_sw else None
    traffic = None
    tp = os.path.join(ROOT, "profiles", "bp_sweep_traffic.json")
    if os.path.exists(tp):
        try:
            traffic = json.load(open(tp)).get("dram_bytes_per_sweep_mixed_16x16_chi16")
        except (OSError, ValueError):
            traffic = None
    line = {
        "metric": METRIC,
        "value": value,
        "unit": "solves/s",
        "n_gpus": world,
        "steps": K,
        "warmup": args.warmup,
        "ms_per_step": res_ms / K,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "mixed: c64 BP sweeps (3xTF32 / FP32 products, FP64 sums; c128 at bonds up to 8) on a c128 state; FP64 absorb, "
                 "truncation, measurement",
        "data": "synthetic (seeded kicked-Ising circuit and Pauli observable)",
        "config": workload_config(theta_h, world),
        "e2e": {"value": e2e_value, "unit": "solves/s", "h2d_bytes_per_step": stats[-1]["h2d"],
                "d2h_bytes_per_step": stats[-1]["d2h"]},
        "gpu_launches": int(launches),
        "observable": {"mixed": [sums[-1].real, sums[-1].imag]},
        "bp_sweeps_per_solve": stats[-1]["sweeps"],
        "wall_s": t_wall,
        "clocks": clk.summary(),
    }
    line["roofline"] = {
        "kernel": "BP sweep (k_pair_absorb_tc + k_pair_gram_tc + k_leg_apply_tc + k_gram_tc + k_msg_finalize + k_segmented_sum, one CUDA graph)",
        "bound": "tensor",
        "achieved": achieved,
        "peak": tf_peak,
        "unit": "TFLOP/s",
        "frac": (achieved / tf_peak) if achieved else None,
        "peak_source": "MEASURED_PEAKS.json bf16_tflops_sustained (of measured)" if peaks else "fallback 1.4 PF/s",
        "traffic": traffic,
        "algorithmic": {"flops_per_sweep": tot_fl / n_sw if n_sw else None,
                        "bytes_per_sweep": tot_by / n_sw if n_sw else None,
                        "sweep_ms": tot_ms / n_sw if n_sw else None,
                        "hbm_achieved_gbs": (tot_by / n_sw) / ((tot_ms / n_sw) / 1e3) / 1e9 if n_sw else None,
                        "hbm_peak_gbs": peaks.get("hbm_gbs")},
    }
    # the DRAM bytes that a sweep moves at D = 32 (counters, scaled: see the
    # file) over the measured sweep time: how close the kernels run to the
    # copy bandwidth on the traffic they must move
    if traffic and n_sw and peaks.get("hbm_gbs"):
        rate = traffic / ((tot_ms / n_sw) / 1e3) / 1e9
        line["roofline"]["schedule_traffic"] = {"gbs": rate, "frac_of_hbm": rate / peaks["hbm_gbs"],
                                                "traffic_over_algorithmic": traffic / (tot_by / n_sw)}
    if not args.no_fp64:
        # one untimed solve per arm first, as the mixed arm's warm-up: the
        # first BP loop of a shape class on a device runs the wave-budget
        # autotuner (a few sweeps per candidate), which is not solve time
        solve(tb, tb.C128, theta_h, pauli_text)
        solve(tb, tb.C64, theta_h, pauli_text)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        s64, st64 = solve(tb, tb.C128, theta_h, pauli_text)
        torch.cuda.synchronize()
        e1.record()
        torch.cuda.synchronize()
        ms64 = e0.elapsed_time(e1)
        line["plain_fp64"] = {"solves_per_s": 1e3 / ms64, "warmup": 1, "observable": [s64.real, s64.imag],
                              "bp_sweeps": st64["sweeps"], "sweep_ms": st64["totals"][0] / max(1, st64["totals"][3])}
        line["dE_vs_fp64"] = abs(sums[-1] - s64)
        line["dterm_max_vs_fp64"] = float(np.max(np.abs(stats[-1]["per"] - st64["per"])))
        # complex64 storage throughout (TNBP_C64): faster, but its rounding
        # of the state each step limits the aggregated observable
        torch.cuda.synchronize()
        e0.record()
        s32, st32 = solve(tb, tb.C64, theta_h, pauli_text)
        e1.record()
        torch.cuda.synchronize()
        line["c64_storage"] = {"solves_per_s": 1e3 / e0.elapsed_time(e1), "warmup": 1, "bp_sweeps": st32["sweeps"],
                               "dE_vs_fp64": abs(s32 - s64),
                               "dterm_max_vs_fp64": float(np.max(np.abs(st32["per"] - st64["per"])))}
        line["speedup_vs_fp64"] = line["plain_fp64"]["solves_per_s"] and e2e_value / line["plain_fp64"]["solves_per_s"]
    if args.served_requests > 0:
        line["served"] = served_summary(tb, args.served_requests)
    if args.config5:
        line["config5_reduced"] = config5_summary(tb)
    if not args.no_fp64:
        line["random_circuit"] = random_circuit_summary(tb)
    if world == 1 and not args.no_cpu:
        # the reference CPU solve and the GPU solves of the same prefix of
        # the workload, timed in this run (apples to apples)
        ref_vals, vm, vp = {}, {}, {}
        cpu_s = cpu_sample(theta_h, values=ref_vals)
        gm, sm = gpu_prefix_solve(tb, tb.MIXED, theta_h, pauli_text, per_term=vm)
        gp, sp = gpu_prefix_solve(tb, tb.C128, theta_h, pauli_text, per_term=vp)

        def term_diff(got):
            if not ref_vals or len(got.get("one", [])) != len(ref_vals["one"]) or \
                    len(got.get("two", [])) != len(ref_vals["two"]):
                return None
            d = [abs(a - b) for a, b in zip(got["one"] + got["two"], ref_vals["one"] + ref_vals["two"])]
            return max(d) if d else 0.0
        if cpu_s is not None:
            line["cpu_baseline"] = {"value": 1.0 / cpu_s, "unit": "solves/s", "cores": os.cpu_count(),
                                    "kind": "reference", "seconds": cpu_s, "sample": prefix_sample_text()}
        line["cpu_matched"] = {
            "sample": prefix_sample_text(),
            "cpu_reference_s": cpu_s, "gpu_mixed_s": gm, "gpu_plain_fp64_s": gp,
            "speedup_mixed": (cpu_s / gm) if cpu_s else None,
            "speedup_plain_fp64": (cpu_s / gp) if cpu_s else None,
            "dE_mixed_vs_plain": abs(sm - sp),
            # the reference app's printed per-term values (16 digits) against
            # the GPU paths' on the same prefix
            "parity_vs_reference": {"terms": len(ref_vals.get("one", [])) + len(ref_vals.get("two", [])),
                                    "max_dterm_plain_fp64": term_diff(vp), "max_dterm_mixed": term_diff(vm)},
            "note": "GPU times through the public API from QASM text (host wall clock, includes TPO build)"}
    print(json.dumps(line))
    if dist:
        dist.destroy_process_group()


def cpu_sample(theta_h, steps=CPU_SAMPLE_STEPS, values=None):
    """One complete solve of the reference's estimator app
    (oracle/_ref/estimator: the unchanged tnbp estimator app and headers on
    the project's CPU tensor backend, OpenMP threads = all host cores) on the
    first `steps` Floquet steps of the same workload (same lattice, angles,
    chi, tolerances and observable; BP at bond dimension <= 16): QASM read,
    TPO built, every step's absorb / BP / truncation, then the Pauli terms.
    Returns the measured wall time of that solve; nothing is extrapolated.
    With a dict `values`, the per-term values the app printed are stored in
    it (keys "one" and "two")."""
    exe = os.path.join(ROOT, "oracle", "_ref", "estimator")
    if not os.path.exists(exe):
        return None
    _, pauli_text = workload()
    d = tempfile.mkdtemp()
    qp, pp = os.path.join(d, "c.qasm"), os.path.join(d, "p.txt")
    open(qp, "w").write(kicked_ising_qasm(steps, THETA_J, theta_h))
    open(pp, "w").write(pauli_text)
    env = dict(os.environ, OMP_NUM_THREADS=str(os.cpu_count()))
    t = time.perf_counter()
    r = subprocess.run([exe, "--circuit", qp, "--sparse_pauli", pp, "--max_bond_dim", str(CHI), "--bp_tolerance",
                        repr(BP_TOL), "--max_bp_iterations", str(BP_MAXIT), "--sv_min", repr(SV_MIN)],
                       check=True, capture_output=True, env=env, timeout=1800, text=True)
    dt = time.perf_counter() - t
    if values is not None:
        values["one"] = [float(v) for v in re.findall(r"single site operator at site \d+ (\S+)", r.stdout)]
        values["two"] = [float(v) for v in re.findall(r"two site operator at sites \(\d+,\d+\) (\S+)", r.stdout)]
    return dt


def prefix_sample_text(steps=CPU_SAMPLE_STEPS):
    return (f"one complete estimator solve of the first {steps} of the {STEPS} Floquet steps of this workload "
            f"(same lattice, angles, chi, tolerances and observable; BP at bond dimension <= 16), wall clock; "
            f"value = those prefix solves per second, measured, not extrapolated to the {STEPS}-step solve")


def gpu_prefix_solve(tb, precision, theta_h, pauli_text, steps=CPU_SAMPLE_STEPS, per_term=None):
    """The same prefix solve as cpu_sample through the public API on the GPU
    (QASM text in, estimator loop, Pauli sum out), host wall clock."""
    import torch
    qasm = kicked_ising_qasm(steps, THETA_J, theta_h)
    torch.cuda.synchronize()
    t = time.perf_counter()
    total, _, _ = estimator_from_qasm(tb, precision, qasm, pauli_text, CHI, per_term=per_term)
    torch.cuda.synchronize()
    return time.perf_counter() - t, total


def run_reference(args, rank, world):
    if rank != 0:
        return
    theta_h, _ = workload()
    exe = os.path.join(ROOT, "oracle", "_ref", "estimator")
    if not os.path.exists(exe):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/estimator is not built (build() compiles "
                                                              "it from the reference tree)"}))
        return
    for _ in range(args.warmup):
        cpu_sample(theta_h)
    times = []
    t_all = time.perf_counter()
    for _ in range(args.steps):
        times.append(cpu_sample(theta_h))
    wall = time.perf_counter() - t_all
    value = len(times) / sum(times)
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": value, "unit": "solves/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * sum(times) / len(times), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "c128", "data": "synthetic (seeded kicked-Ising circuit and Pauli observable)",
        "config": workload_config(theta_h, world),
        "sample": prefix_sample_text(),
        "wall_s": wall,
        "cpu_baseline": {"value": value, "unit": "solves/s", "cores": os.cpu_count(), "kind": "reference",
                         "sample": prefix_sample_text()},
        "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def main():
    global L_SIDE, STEPS
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--served-requests", type=int, default=SERVED_N,
                    help="requests of the served stream to run (0 skips the served leg)")
    ap.add_argument("--served-only", action="store_true",
                    help="run only the served leg and print its summary as one JSON line")
    ap.add_argument("--config5", action="store_true",
                    help="also run the 32x32 large solve at chi 16 (both paths; several minutes)")
    ap.add_argument("--config5-only", action="store_true",
                    help="run only the 32x32 large solve at chi 16 and print its summary as one JSON line")
    ap.add_argument("--lattice", type=int, default=L_SIDE,
                    help="lattice side (default 16; smaller sides are for profiling captures only)")
    ap.add_argument("--nsteps", type=int, default=STEPS,
                    help="Floquet steps per solve (default 20; fewer only for profiling captures)")
    args = ap.parse_args()
    L_SIDE, STEPS = args.lattice, args.nsteps
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", str(args.gpus if args.gpus == 1 else 1)))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.config5_only:
        import tnbp_b200 as tb
        if rank == 0:
            print(json.dumps({"config5_reduced": config5_summary(tb)}))
    elif args.served_only:
        import tnbp_b200 as tb
        if rank == 0:
            print(json.dumps({"served": served_summary(tb, args.served_requests)}))
    elif args.impl == "reference":
        run_reference(args, rank, world)
    else:
        run_ours(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
