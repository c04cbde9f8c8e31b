"""AbsorbTPO's site kernel at the shapes where its blocks change: fewer and more
than 256 bond indices per site (one index: 256 threads share the operator's
elements), more than 128 operator elements, ranks of 1 and odd ranks, another
physical dimension than 2, and the complex64 copy that a mixed job writes
along (read by the sweep after it, and again after a site was replaced).

Site tensors against the numpy oracle at the 1e-13 of the other AbsorbTPO
tests (complex64 storage: two roundings of 2^-24 and sums of two products,
1e-6); the mixed job's messages at the 5e-5 of the reduced-precision tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

CASES = [((1, 1, 1), (2, 3, 4), 2), ((5, 2), (3, 1), 2), ((7, 6, 8), (2, 2, 2), 2), ((16, 17), (4, 5), 2), ((3, 3, 3, 3), (4, 3, 2, 5), 2),
         ((4, 3), (2, 3), 3), ((300,), (2,), 2)]


def _setup(dims, ranks, d):
    rng = np.random.default_rng(sum(dims) + sum(ranks))
    edges = [(0, k + 1) for k in range(len(dims))]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    sites = bn.sites_of(edges)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [d]) for s in sites]
    V = [v / np.linalg.norm(v) for v in V]
    E = []
    for m in range(2 * len(edges)):
        A = gauss((dims[m % len(edges)],) * 2)
        M = A @ A.conj().T
        E.append(M / np.linalg.norm(M))
    ops = [gauss([ranks[m] for m in bn.bonds_of(edges, s)] + [d, d]) / 2 for s in sites]
    return edges, V, E, ops


def _layer(edges, ops, d):
    rank = [ops[0].shape[k] for k in range(len(edges))]
    off, data, o = [], [], 0
    for x in ops:
        off.append(o)
        data.append(np.asarray(x, np.complex128).reshape(-1, order="F"))
        o += x.size
    return tb.TPOLayer(rank, off, np.concatenate(data))


@pytest.mark.parametrize("prec,tol", [(tb.C128, 1e-13), (tb.C64, 1e-6)], ids=["c128", "c64"])
@pytest.mark.parametrize("dims,ranks,d", CASES, ids=["x".join(map(str, c[0])) + "-d%d" % c[2] for c in CASES])
def test_absorbed_sites_match_oracle(dims, ranks, d, prec, tol):
    edges, V, E, ops = _setup(dims, ranks, d)
    want, _ = bn.absorb_tpo(edges, V, E, ops)
    with tb.State(edges, prec, pdims=[d] * len(V)) as st:
        st.set_state(V, E)
        tb.AbsorbTPO(st, _layer(edges, ops, d))
        for s, w in enumerate(want):
            assert np.max(np.abs(st.get_site(s) - w)) <= tol


def test_mixed_sweep_reads_the_copy_written_along():
    edges, V, E, ops = _setup((7, 6, 8), (2, 2, 2), 2)
    V1, E1 = bn.absorb_tpo(edges, V, E, ops)
    V2 = [v[..., ::-1].copy() for v in V1]
    with tb.State(edges, tb.MIXED) as st:
        st.set_state(V, E)
        tb.AbsorbTPO(st, _layer(edges, ops, 2))
        for state in (V1, V2):  # as absorbed, then with replaced sites
            if state is V2:
                st.set_state(V2, E1)
            tb.BeliefPropagation(st)
            F = bn.bp_sweep(edges, state, E1)
            assert max(float(np.max(np.abs(st.get_message(m) - F[m]))) for m in range(2 * len(edges))) <= 5e-5
