"""What the framework's speed is measured on: whole estimator solves, single
Floquet steps, loops of BP sweeps, cluster measurements and served batches,
through the Python entry points of tnbp_b200, from calls of a few
milliseconds to lattices whose tensors fill gigabytes.

A case is a dict of plain values.  `kind` says which path it runs:
  estimator  a kicked-Ising program from |0...0>: every Floquet step absorbs
             the layer, runs the BP loop and truncates; then all Z and all
             nearest-neighbour ZZ are measured
  circuit    the same from OpenQASM text of a random U3 + CZ circuit with a
             random Pauli observable
  floquet    one more Floquet step (absorb, BP at twice chi, truncate) of a
             state that is already at chi, and its observables
  bp         a fixed number of BP sweeps on a state of given bond dimensions;
             the messages are read back
  cluster    Pauli strings of several qubits measured on their clusters
  served     a batch of kicked-Ising requests through the server

`exact` computes the same in complex128 with torch, from the definitions.
Values of the reduced-precision paths (their sweeps carry 32-bit numbers) are
returned as complex64, those of the complex128 path as complex128.  Truncated
site tensors are defined up to a phase (or a rotation) per bond, so a step's
new state is returned as what it is kept for: the expectation values on every
site and every bond, beside the kept dimensions.  (The discarded weights are
squares of singular values near the messages' rounding, sure to fewer digits
than the values are.)
"""
import math

import numpy as np
import torch

import tnbp_b200 as tb

PRECISION = {"c128": tb.C128, "mixed": tb.MIXED, "c64": tb.C64}
SV_MIN = 1e-8
BP_TOL = 1e-8
BP_MAX = 50
FLOQUET_SWEEPS = 3  # BP iterations of one step; the kicked-Ising solves take 3 to 4


def listed():
    return [
        # the smallest solve: launches and host latency
        dict(name="estimator-4x4-chi4-c128", kind="estimator", nx=4, ny=4, chi=4, steps=5, precision="c128"),
        # small lattice at a working chi, reduced precision
        dict(name="estimator-6x5-chi8-mixed", kind="estimator", nx=6, ny=5, chi=8, steps=6, precision="mixed"),
        # the random-circuit estimator from text, bonds up to 8
        dict(name="circuit-10x10-mixed", kind="circuit", nx=10, ny=10, layers=12, chi=32, precision="mixed"),
        # sweeps at the bond dimension of chi = 16 solves
        dict(name="bp-8x8-d32-mixed", kind="bp", nx=8, ny=8, dims="4,4,2", ragged=False, sweeps=6, precision="mixed"),
        # every bond another dimension, odd ones among them
        dict(name="bp-7x5-ragged-mixed", kind="bp", nx=7, ny=5, dims="6,5", ragged=True, sweeps=6, precision="mixed"),
        dict(name="bp-7x6-ragged-c128", kind="bp", nx=7, ny=6, dims="6,4", ragged=True, sweeps=4, precision="c128"),
        # complex64 storage
        dict(name="bp-6x6-d16-c64", kind="bp", nx=6, ny=6, dims="4,4", ragged=False, sweeps=8, precision="c64"),
        # one step of the large kicked-Ising solves, both paths
        dict(name="floquet-12x12-chi16-mixed", kind="floquet", nx=12, ny=12, chi=16, precision="mixed"),
        dict(name="floquet-8x8-chi16-c128", kind="floquet", nx=8, ny=8, chi=16, precision="c128"),
        # chi = 32 requests: BP at D = 64
        dict(name="floquet-5x5-chi32-mixed", kind="floquet", nx=5, ny=5, chi=32, precision="mixed"),
        # Pauli strings on several qubits
        dict(name="cluster-6x6-d16-c128", kind="cluster", nx=6, ny=6, dims="4,4", ragged=False, terms=12, precision="c128"),
        # requests that share the server's sweeps
        dict(name="served-12-mixed", kind="served", requests=12, side_lo=4, side_hi=6, chi=8, depth_lo=4, depth_hi=7,
             precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["estimator", "circuit", "floquet", "floquet", "bp", "bp", "bp", "cluster", "served"])
    prec = rng.choice(["mixed", "mixed", "c128", "c64"])
    nx, ny = rng.randint(3, 9), rng.randint(3, 9)
    if kind == "estimator":
        chi = _log_int(rng, 2, 16)
        return dict(kind=kind, nx=min(nx, 7), ny=min(ny, 7), chi=chi, steps=rng.randint(3, 7), precision=rng.choice(["c128", "mixed"]))
    if kind == "circuit":
        return dict(kind=kind, nx=nx, ny=ny, layers=rng.randint(4, 12), chi=32, precision=rng.choice(["c128", "mixed"]))
    if kind == "floquet":
        chi = _log_int(rng, 4, 24)
        if chi > 16:
            nx, ny = min(nx, 4), min(ny, 5)
        return dict(kind=kind, nx=nx, ny=ny, chi=chi, precision=rng.choice(["c128", "mixed"]))
    if kind == "served":
        lo = rng.randint(4, 5)
        return dict(kind=kind, requests=rng.randint(2, 12), side_lo=lo, side_hi=rng.randint(lo, 6), chi=rng.choice([4, 8]),
                    depth_lo=3, depth_hi=rng.randint(4, 6), precision=rng.choice(["mixed", "mixed", "c128"]))
    r = [_log_int(rng, 2, 6), _log_int(rng, 2, 6)]
    if r[0] * r[1] > 24:
        nx, ny = min(nx, 6), min(ny, 6)
    case = dict(kind=kind, nx=nx, ny=ny, dims="%d,%d" % tuple(r), ragged=rng.random() < 0.5)
    if kind == "cluster":
        return dict(case, nx=max(4, min(nx, 6)), ny=max(4, min(ny, 6)), dims="%d,%d" % (min(r[0], 4), min(r[1], 4)),
                    terms=rng.randint(2, 16), precision="c128")
    return dict(case, sweeps=rng.randint(2, 8), precision=prec)


# ------------------------------------------------------------------ inputs
def _lattice(nx, ny):
    """Open square lattice, site x + nx y: bonds of a site to the right, then up."""
    edges = []
    for s in range(nx * ny):
        if s % nx + 1 < nx:
            edges.append((s, s + 1))
        if s + nx < nx * ny:
            edges.append((s, s + nx))
    return edges


def _bonds(edges, n):
    legs = [[] for _ in range(n)]
    for m, (a, b) in enumerate(edges):
        legs[a].append(m)
        legs[b].append(m)
    return legs


def _angles(seed):
    rng = np.random.default_rng([seed, 1])
    # the regime in which loopy BP converges on these lattices
    return float(rng.uniform(-0.85, -0.72)), float(rng.uniform(0.25, 0.45))


def _z_and_zz(edges, n):
    """(qubits, letters, coefficient) of every Z and every nearest-neighbour ZZ."""
    return [((i,), "Z", 1.0 / n) for i in range(n)] + [((a, b), "ZZ", 1.0) for a, b in edges]


def _pauli_text(terms, n):
    lines = []
    for qubits, letters, c in terms:
        chars = ["I"] * n
        for q, l in zip(qubits, letters):
            chars[n - 1 - q] = l
        lines.append("%r %s" % (c, "".join(chars)))
    return "\n".join(lines) + "\n"


def _random_terms(rng, edges, n, count):
    terms = []
    for k in range(count):
        l = [str(x) for x in rng.choice(list("XYZ"), size=2)]
        if k % 2:
            a, b = edges[int(rng.integers(len(edges)))]
            terms.append(((a, b), l[0] + l[1], float(rng.normal())))
        else:
            terms.append(((int(rng.integers(n)),), l[0], float(rng.normal())))
    return terms


def _line_terms(rng, nx, ny, count):
    """Pauli strings of 2 to 4 qubits along one row: one shortest path joins them."""
    terms = []
    for _ in range(count):
        y, k = int(rng.integers(ny)), int(rng.integers(2, 5))
        xs = sorted(int(x) for x in rng.choice(nx, size=min(k, nx), replace=False))
        if len(xs) == 2 and xs[1] == xs[0] + 1:
            xs = [0, nx - 1]
        terms.append(([x + nx * y for x in xs], "".join(str(c) for c in rng.choice(list("XYZ"), size=len(xs)))))
    return terms


def _layers(case, seed):
    """Operator layers whose bonds multiply up to the case's bond dimensions;
    each operator bond's weights decay, as a gate's Schmidt values do.  A
    ragged lattice's dimensions belong to the case, its numbers to the seed."""
    edges, n = _lattice(case["nx"], case["ny"]), case["nx"] * case["ny"]
    legs = _bonds(edges, n)
    rng, shape = np.random.default_rng([seed, 2]), np.random.default_rng([case["nx"], case["ny"]])
    out = []
    for top in (int(x) for x in case["dims"].split(",")):
        rank = shape.integers(1 if out else 2, top + 1, size=len(edges)) if case["ragged"] else np.full(len(edges), top)
        ops = []
        for s in range(n):
            sh = [int(rank[m]) for m in legs[s]] + [2, 2]
            o = rng.normal(size=sh) + 1j * rng.normal(size=sh)
            for k in range(len(legs[s])):
                o *= (0.7 ** np.arange(sh[k])).reshape([-1 if j == k else 1 for j in range(len(sh))])
            ops.append(o / np.sqrt(8.0))
        out.append(ops)
    return edges, n, out


def _circuit(case, seed):
    """(gates by layer, qasm text, terms): U3 on every qubit, CZ on one of four colourings, a barrier."""
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    rng = np.random.default_rng([seed, 3])
    layers, text = [], ["OPENQASM 2.0;", 'include "qelib1.inc";', "qreg q[%d];" % n]
    for t in range(case["layers"]):
        u = rng.uniform(0.0, 2 * math.pi, size=(n, 3))
        cz = []
        for s in range(n):
            x, y = s % nx, s // nx
            if t % 4 < 2 and x % 2 == t % 4 and x + 1 < nx:
                cz.append((s, s + 1))
            if t % 4 >= 2 and y % 2 == t % 4 - 2 and y + 1 < ny:
                cz.append((s, s + nx))
        layers.append((u, cz))
        text += ["u3(%r,%r,%r) q[%d];" % (*map(float, u[s]), s) for s in range(n)]
        text += ["cz q[%d],q[%d];" % e for e in cz] + ["barrier q;"]
    edges = sorted({e for _, cz in layers for e in cz})
    return layers, edges, "\n".join(text) + "\n", _random_terms(rng, edges, n, 48)


def _requests(case, seed):
    rng = np.random.default_rng([seed, 4])
    out = []
    for _ in range(case["requests"]):
        L = int(rng.integers(case["side_lo"], case["side_hi"] + 1))
        edges = _lattice(L, L)
        out.append(dict(L=L, steps=int(rng.integers(case["depth_lo"], case["depth_hi"] + 1)), theta_j=-math.pi / 4,
                        theta_h=float(rng.uniform(0.25, 0.45)), terms=_random_terms(rng, edges, L * L, 8)))
    return out


def _kicked_ising(edges, theta_j, theta_h):
    # RZZ(theta) = exp(-i theta/2 ZZ), RX(theta) = exp(-i theta/2 X)
    return tb.KickedIsingTPO(edges, theta_j / 2.0, 0.0, theta_h / 2.0, 1.0)


def prepare(case, seed):
    kind, prec = case["kind"], PRECISION[case["precision"]]
    if kind == "circuit":
        _, _, text, terms = _circuit(case, seed)
        n = case["nx"] * case["ny"]
        return dict(case=case, qasm=text, pauli=_pauli_text(terms, n))
    if kind == "served":
        reqs = []
        for r in _requests(case, seed):
            edges = tb.bond_square_lattice(r["L"], r["L"])
            reqs.append((r, tb.load_sparse_pauli(_pauli_text(r["terms"], r["L"] * r["L"]), edges)))
        return dict(case=case, server=tb.Server(prec, max_active=64), requests=reqs)
    nx, ny = case["nx"], case["ny"]
    edges, n = _lattice(nx, ny), nx * ny
    if kind in ("bp", "cluster"):
        _, _, layers = _layers(case, seed)
        st = tb.InitTensorProductState(edges, prec)
        for ops in layers:
            tb.AbsorbTPO(st, tb.TPOLayer.from_ops(edges, ops))
        if kind == "cluster":
            for _ in range(4):
                tb.BeliefPropagation(st)
            return dict(case=case, state=st, terms=_line_terms(np.random.default_rng([seed, 5]), nx, ny, case["terms"]))
        return dict(case=case, state=st)
    theta_j, theta_h = _angles(seed)
    terms = tb.load_sparse_pauli(_pauli_text(_z_and_zz(edges, n), n), edges)
    layer = _kicked_ising(edges, theta_j, theta_h)
    if kind == "estimator":
        return dict(case=case, edges=edges, layer=layer, terms=terms)
    st = tb.InitTensorProductState(edges, prec)
    handle = st.tpo(layer)
    for _ in range(_steps_to(case["chi"])):
        tb.AbsorbTPO(st, handle)
        tb.BeliefPropagationLoop(st, BP_TOL, FLOQUET_SWEEPS)
        tb.Truncation(st, case["chi"], SV_MIN)
    return dict(case=case, state=st, layer=handle, terms=terms)


def _steps_to(chi):
    """Floquet steps after which every bond holds chi singular values: they
    double at most, and the smallest only grow above the cut after some more."""
    return math.ceil(math.log2(chi)) + 4


def _values(case, per, terms):
    """Values in the observable's row order, at the path's precision."""
    v = np.asarray(per)[np.argsort(np.asarray(terms.row), kind="stable")]
    return _at(case, v)


def _at(case, v):
    return v if case["precision"] == "c128" else v.astype(np.complex64)


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind, prec = case["kind"], PRECISION[case["precision"]]
    if kind == "estimator":
        with tb.InitTensorProductState(state["edges"], prec) as st:
            layer = st.tpo(state["layer"])
            for _ in range(case["steps"]):
                tb.AbsorbTPO(st, layer)
                tb.BeliefPropagationLoop(st, BP_TOL, BP_MAX)
                tb.Truncation(st, case["chi"], SV_MIN)
            total, per = tb.MeasurePauliSum(st, state["terms"])
        return dict(total=_at(case, np.array([total])), values=_values(case, per, state["terms"]))
    if kind == "circuit":
        edges = tb.EdgesFromQasm(state["qasm"])
        terms = tb.load_sparse_pauli(state["pauli"], edges)
        with tb.InitTensorProductState(edges, prec) as st:
            for layer in tb.QasmToTPO(state["qasm"], edges):
                tb.AbsorbTPO(st, layer)
                tb.BeliefPropagationLoop(st, BP_TOL, BP_MAX)
                tb.Truncation(st, case["chi"], SV_MIN)
            total, per = tb.MeasurePauliSum(st, terms)
        return dict(total=_at(case, np.array([total])), values=_values(case, per, terms))
    if kind == "floquet":
        st = state["state"]
        tb.AbsorbTPO(st, state["layer"])
        tb.BeliefPropagationLoop(st, BP_TOL, FLOQUET_SWEEPS)
        dims, _ = tb.Truncation(st, case["chi"], SV_MIN)
        total, per = tb.MeasurePauliSum(st, state["terms"])
        return dict(total=_at(case, np.array([total])), values=_values(case, per, state["terms"]), dims=dims)
    if kind == "bp":
        st = state["state"]
        for _ in range(case["sweeps"]):
            tb.BeliefPropagation(st)
        return _at(case, np.concatenate([e.reshape(-1, order="F") for e in st.get_E()]))
    if kind == "cluster":
        return _at(case, tb.MeasureCluster(state["state"], state["terms"])[0])
    server = state["server"]
    ids = [server.submit_kicked_ising(r["L"], case["chi"], r["steps"], r["theta_j"], r["theta_h"], terms)
           for r, terms in state["requests"]]
    while True:
        active, queued, _ = server.step()
        if active == 0 and queued == 0:
            break
    return _at(case, np.array([server.result(i) for i in ids]))


# -------------------------------------------------------------------- work
def _tree(g):
    """Leg contractions of a degree-g site whose targets share partial products."""
    return 0 if g < 2 else g + _tree(g // 2) + _tree(g - g // 2)


def _sweep_work(edges, n, dim, elem):
    """Bytes and flops of one BP sweep at bond dimensions dim[m]."""
    byts = flops = 0.0
    for legs in _bonds(edges, n):
        size = 2.0 * math.prod(dim[m] for m in legs)
        mean = sum(dim[m] for m in legs) / len(legs)
        byts += size * elem
        flops += 8.0 * size * mean * (_tree(len(legs)) + len(legs))
    return byts + 4.0 * sum(d * d for d in dim) * 16, flops


def _state_bytes(edges, n, dim, elem):
    return sum(2.0 * elem * math.prod(dim[m] for m in legs) for legs in _bonds(edges, n))


def _step_work(edges, n, old, chi, sweeps, precision):
    """One Floquet step from bond dimension `old` to min(2 old, chi)."""
    big = [2 * old] * len(edges)
    new = [min(2 * old, chi)] * len(edges)
    elem = 8 if precision == "c64" else 16
    sweep = _sweep_work(edges, n, big, 16 if precision == "c128" else 8)
    byts = _state_bytes(edges, n, [old] * len(edges), elem) + 2 * _state_bytes(edges, n, big, elem)
    byts += _state_bytes(edges, n, new, elem) + sweeps * sweep[0]
    chain = 0.0  # projecting every leg, the first at full size
    for legs in _bonds(edges, n):
        size = 2.0 * (2 * old) ** len(legs)
        for k in range(len(legs)):
            chain += 8.0 * size * new[0] * (new[0] / (2.0 * old)) ** k
    return byts, sweeps * sweep[1] + chain


def work(case):
    kind, prec = case["kind"], case["precision"]
    if kind == "served":
        side = 0.5 * (case["side_lo"] + case["side_hi"])
        edges, n = _lattice(round(side), round(side)), round(side) ** 2
        steps, chi, times = round(0.5 * (case["depth_lo"] + case["depth_hi"])), case["chi"], case["requests"]
    else:
        edges, n, times = _lattice(case["nx"], case["ny"]), case["nx"] * case["ny"], 1
    if kind in ("bp", "cluster"):
        elem = 16 if prec == "c128" else 8
        tops = [int(x) for x in case["dims"].split(",")]
        mid = math.prod((t + (1 if i else 2)) / 2.0 for i, t in enumerate(tops)) if case["ragged"] else math.prod(tops)
        byts, flops = _sweep_work(edges, n, [mid] * len(edges), elem)
        if kind == "bp":
            return dict(bytes=case["sweeps"] * byts, flops=case["sweeps"] * flops)
        # per term about half a row of sites, each with its legs absorbed and one Gram of d D columns
        size = 2.0 * mid**4
        sites = case["terms"] * case["nx"] / 2.0
        return dict(bytes=sites * size * elem, flops=2 * sites * 8.0 * size * mid * 5)
    if kind == "floquet":
        byts, flops = _step_work(edges, n, case["chi"], case["chi"], FLOQUET_SWEEPS, prec)
        return dict(bytes=byts, flops=flops)
    byts = flops = 0.0
    if kind == "circuit":
        for t in range(case["layers"]):
            b, f = _step_work(edges, n, 2 ** min(2, t // 4), 32, 2, prec)
            byts, flops = byts + b / 4, flops + f / 4  # a layer's gates touch a quarter of the bonds
    else:
        chi = case["chi"]
        for t in range(case["steps"] if kind == "estimator" else steps):
            b, f = _step_work(edges, n, min(2**t, chi), chi, 3, prec)
            byts, flops = byts + b, flops + f
    return dict(bytes=times * byts, flops=times * flops)


# ------------------------------------------------------------------- exact
class _Exact:
    """The PEPS, its messages and the steps on them in complex128 with torch."""

    def __init__(self, edges, n):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.edges, self.n, self.legs = edges, n, _bonds(edges, n)
        self.V = []
        for legs in self.legs:
            v = torch.zeros([1] * len(legs) + [2], dtype=torch.complex128, device=self.dev)
            v[..., 0] = 1.0
            self.V.append(v)
        self.E = [torch.ones(1, 1, dtype=torch.complex128, device=self.dev) for _ in range(2 * len(edges))]

    def tensor(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.complex128)).to(self.dev)

    def incoming(self, s, m):
        return self.E[m + len(self.edges)] if self.edges[m][0] == s else self.E[m]

    def absorb(self, ops, rank):
        """V'[.., v + D o, .., q] = sum_p O[.., o, .., p, q] V[.., v, .., p]; messages get the identity on o."""
        for s, legs in enumerate(self.legs):
            g, v, o = len(legs), self.V[s], self.tensor(ops[s])
            t = torch.tensordot(v, o, dims=([g], [g]))  # v.., o.., q
            order = [x for k in range(g) for x in (g + k, k)] + [2 * g]
            self.V[s] = t.permute(order).reshape([v.shape[k] * o.shape[k] for k in range(g)] + [2]).contiguous()
        for m in range(2 * len(self.edges)):
            eye = torch.eye(int(rank[m % len(self.edges)]), dtype=torch.complex128, device=self.dev)
            self.E[m] = torch.kron(eye, self.E[m])

    @staticmethod
    def on_leg(t, k, mat):
        return torch.movedim(torch.tensordot(t, mat, dims=([k], [0])), -1, k)

    @staticmethod
    def gram(a, b, keep):
        """N[c, c'] = sum a[.., c, ..] conj(b[.., c', ..]) over every other index."""
        rest = [i for i in range(a.dim()) if i not in keep]
        return torch.tensordot(a, b.conj(), dims=(rest, rest))

    def sweep(self):
        new = [None] * len(self.E)
        for s, legs in enumerate(self.legs):
            for k, m in enumerate(legs):
                t = self.V[s]
                for j, q in enumerate(legs):
                    if j != k:
                        t = self.on_leg(t, j, self.incoming(s, q))
                x = self.gram(t, self.V[s], [k])
                new[m if self.edges[m][0] == s else m + len(self.edges)] = x / torch.linalg.norm(x)
        dist = sum(float(torch.linalg.norm(a - b / torch.linalg.norm(b))) for a, b in zip(new, self.E))
        self.E = new
        return dist / len(new)

    def loop(self, tol, most):
        """Sweeps until the next one would move the messages by less than tol, at most `most`."""
        if most <= 0:
            return
        self.sweep()
        done = 1
        while True:
            kept = self.E
            dist = self.sweep()
            if dist < tol or done >= most:
                self.E = kept  # the last sweep only measures the distance
                return
            done += 1

    @staticmethod
    def root(m):
        u, s, vh = torch.linalg.svd(m)
        keep = s > SV_MIN
        sq = torch.sqrt(torch.where(keep, s, torch.zeros_like(s)))
        inv = torch.where(sq > math.sqrt(SV_MIN), 1.0 / torch.where(sq > 0, sq, torch.ones_like(sq)), torch.zeros_like(sq))
        r = (u * sq) @ vh
        return r, (vh.mH * inv) @ u.mH

    def truncate(self, chi):
        ne = len(self.edges)
        pa, pb = [], []
        for m in range(ne):
            ra, sa = self.root(self.E[m])
            rb, sb = self.root(self.E[m + ne])
            t = ra.T @ rb
            x, s, y = torch.linalg.svd(t / torch.linalg.norm(t))
            k = max(1, min(chi, int((s > SV_MIN).sum())))
            rt = torch.sqrt(s[:k])
            pa.append(sa.T @ (x[:, :k] * rt))
            pb.append(((rt[:, None] * y[:k]) @ sb).T)
            self.E[m] = self.E[m + ne] = torch.diag(s[:k]).to(torch.complex128)
        for s, legs in enumerate(self.legs):
            v = self.V[s]
            for k, m in enumerate(legs):
                v = self.on_leg(v, k, pa[m] if self.edges[m][0] == s else pb[m])
            self.V[s] = v / torch.linalg.norm(v)

    def env(self, s, keep, mats=None):
        """sum_x W[x, (t,) p] conj(V[x, (t',) p']): every bond but `keep` closed by its message (or by mats[bond])."""
        legs, t = self.legs[s], self.V[s]
        for k, m in enumerate(legs):
            if m != keep:
                t = self.on_leg(t, k, (mats or {}).get(m, self.incoming(s, m)))
        return self.gram(t, self.V[s], [k for k, m in enumerate(legs) if m == keep] + [len(legs)])

    def pauli(self, letter):
        return self.tensor({"I": [[1, 0], [0, 1]], "X": [[0, 1], [1, 0]], "Y": [[0, -1j], [1j, 0]], "Z": [[1, 0], [0, -1]]}[letter])

    def value(self, qubits, letters):
        if len(qubits) == 1:
            rho = self.env(qubits[0], None)  # p, p'
            return complex((rho * self.pauli(letters).T).sum() / torch.trace(rho))
        a, b = qubits
        m = self.edges.index((a, b)) if (a, b) in self.edges else self.edges.index((b, a))
        ea, eb = self.env(a, m), self.env(b, m)  # t, p, t', p'
        pick = lambda e, o: torch.einsum("tpuq,qp->tu", e, o)
        one = self.pauli("I")
        num = (pick(ea, self.pauli(letters[0])) * pick(eb, self.pauli(letters[1]))).sum()
        return complex(num / (pick(ea, one) * pick(eb, one)).sum())

    def line(self, qubits, letters):
        """A Pauli string along one row, its sites between the first and the last qubit contracted exactly."""
        z = []
        at = dict(zip(qubits, letters))
        path = list(range(qubits[0], qubits[-1] + 1))
        for on in (True, False):
            x = None
            for i in range(len(path) - 1, -1, -1):
                s = path[i]
                right = self.edges.index((s, s + 1)) if i + 1 < len(path) else None
                left = self.edges.index((path[i - 1], s)) if i > 0 else None
                op = self.pauli(at.get(s, "I") if on else "I")
                if i > 0:
                    x = torch.einsum("tpuq,qp->tu", self.env(s, left, {right: x} if x is not None else None), op)
                else:
                    x = (x * torch.einsum("tpuq,qp->tu", self.env(s, right), op)).sum()
            z.append(complex(x))
        return z[0] / z[1]

    def measured(self, terms):
        v = np.array([self.value(q, l) for q, l, _ in terms])
        return dict(total=np.array([sum(c * x for (_, _, c), x in zip(terms, v))]), values=v)


def _ising_ops(ex, theta_j, theta_h):
    """RX(theta_h) after RZZ(theta_j) on every edge: operator bonds of dimension 2."""
    c, s = math.cos(theta_j / 2), -1j * math.sin(theta_j / 2)
    w = [np.diag([np.sqrt(c + 0j)] * 2), np.sqrt(s) * np.diag([1.0, -1.0])]
    rx = np.array([[math.cos(theta_h / 2), -1j * math.sin(theta_h / 2)], [-1j * math.sin(theta_h / 2), math.cos(theta_h / 2)]])
    ops = []
    for legs in ex.legs:
        o = np.zeros([2] * len(legs) + [2, 2], complex)
        for idx in np.ndindex(*[2] * len(legs)):
            m = rx
            for i in idx:
                m = m @ w[i]
            o[idx] = m.T  # [p, q]: q the output
        ops.append(o)
    return ops, [2] * len(ex.edges)


def _exact_ising(edges, n, theta_j, theta_h, steps, chi, most):
    ex = _Exact(edges, n)
    ops, rank = _ising_ops(ex, theta_j, theta_h)
    for _ in range(steps):
        ex.absorb(ops, rank)
        ex.loop(BP_TOL, most)
        ex.truncate(chi)
    return ex


def _exact_circuit(case, seed):
    layers, edges, _, terms = _circuit(case, seed)
    ex = _Exact(edges, case["nx"] * case["ny"])
    for u, cz in layers:
        rank = [2 if e in cz else 1 for e in edges]
        ops = []
        for s, legs in enumerate(ex.legs):
            th, ph, la = u[s]
            m = np.array([[math.cos(th / 2), -np.exp(1j * la) * math.sin(th / 2)],
                          [np.exp(1j * ph) * math.sin(th / 2), np.exp(1j * (ph + la)) * math.cos(th / 2)]])
            o = np.zeros([rank[b] for b in legs] + [2, 2], complex)
            for idx in np.ndindex(*o.shape[:-2]):
                x = m
                for i, b in zip(idx, legs):
                    if rank[b] == 2:  # CZ = |0><0| I + |1><1| Z
                        x = (np.diag([1.0 - i, float(i)]) if edges[b][0] == s else np.diag([1.0, 1.0 - 2 * i])) @ x
                o[idx] = x.T
            ops.append(o)
        ex.absorb(ops, rank)
        ex.loop(BP_TOL, BP_MAX)
        ex.truncate(case["chi"])
    return ex.measured(terms)


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        return _exact_circuit(case, seed)
    if kind == "served":
        out = []
        for r in _requests(case, seed):
            edges, n = _lattice(r["L"], r["L"]), r["L"] ** 2
            ex = _exact_ising(edges, n, r["theta_j"], r["theta_h"], r["steps"], case["chi"], BP_MAX)
            out.append(ex.measured(r["terms"])["total"][0])
        return np.array(out)
    edges, n = _lattice(case["nx"], case["ny"]), case["nx"] * case["ny"]
    if kind in ("bp", "cluster"):
        _, _, layers = _layers(case, seed)
        ex = _Exact(edges, n)
        for ops in layers:
            rank = [ops[a].shape[ex.legs[a].index(m)] for m, (a, _) in enumerate(edges)]
            ex.absorb(ops, rank)
        for _ in range(case["sweeps"] if kind == "bp" else 4):
            ex.sweep()
        if kind == "bp":
            return np.concatenate([e.T.reshape(-1).cpu().numpy() for e in ex.E])
        terms = _line_terms(np.random.default_rng([seed, 5]), case["nx"], case["ny"], case["terms"])
        return np.array([ex.line(q, l) for q, l in terms])
    theta_j, theta_h = _angles(seed)
    terms = _z_and_zz(edges, n)
    if kind == "estimator":
        ex = _exact_ising(edges, n, theta_j, theta_h, case["steps"], case["chi"], BP_MAX)
        return ex.measured(terms)
    ex = _exact_ising(edges, n, theta_j, theta_h, _steps_to(case["chi"]) + 1, case["chi"], FLOQUET_SWEEPS)
    return dict(ex.measured(terms), dims=None)
