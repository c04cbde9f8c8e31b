"""Precision of the 33- to 64-wide kernels (tc_leg64.cuh, tc_gram64.cuh):
every message of a site is within 1e-6 (Frobenius norm) of the numpy oracle's,
and far closer than a kernel that loses the lo parts of its operands, in the
legs or in the Gram alone, could come (computed beside it).

A message has norm 1.  Up to four stages round to 24 bits or split to as many
(2^-23 of a product at most), with signs that do not agree: a few 2^-23, and
1e-6 is eight of them.  Operands of 11 bits leave 7e-6 or more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

DIMS = [(64, 64), (33, 40), (64, 3, 33), (2, 64, 48), (31, 37, 5), (5, 60, 7, 3), (32, 41, 6), (8, 64, 34, 2), (63, 2, 2, 2), (3, 3, 64, 11),
        (50, 3), (34, 7, 3), (42, 38, 35), (6, 9, 34, 2)]


def tf32(a):
    """Rounded to 11 significant bits."""
    def part(x):
        bits = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
        return ((bits + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32).astype(np.float64)
    return part(a.real) + 1j * part(a.imag)


def message(V, E, k, legs, gram):
    """Message k of the centre with its operands rounded by `legs` and `gram`."""
    g = len(E) // 2
    t = V
    for j in range(g):
        if j != k:
            t = np.moveaxis(np.tensordot(legs(t), legs(E[j + g]), axes=([j], [0])), -1, j)
    rest = [i for i in range(g + 1) if i != k]
    return bn.normalize(np.tensordot(gram(t), gram(V).conj(), axes=(rest, rest)))[0]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_wide_messages_keep_the_lo_parts(dims, prec):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    rng = np.random.default_rng(sum(dims))
    ne = len(dims)
    edges = [(0, k + 1) for k in range(ne)]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = []
    for m in range(2 * ne):
        A = gauss((dims[m % ne],) * 2)
        M = A @ A.conj().T
        E.append(M / np.linalg.norm(M))
    F = bn.bp_sweep(edges, V, E)
    whole = lambda x: x
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        tb.BeliefPropagation(st)
        for k in range(ne):
            assert np.linalg.norm(st.get_message(k) - F[k]) <= 1e-6
            for legs, gram in ((tf32, whole), (whole, tf32)):
                assert np.linalg.norm(message(V[0], E, k, legs, gram) - F[k]) >= 5e-6
