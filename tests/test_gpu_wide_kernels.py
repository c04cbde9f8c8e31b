"""The 33- to 64-wide kernels of the reduced-precision sweeps (tc_leg64.cuh,
tc_gram64.cuh) against the numpy oracle, where their tiles end: leg strides of
1, small and odd (whole-block tiles up to 32), 33 and above, K halves that are
unequal or empty, dimensions that are not multiples of 8 or 4, last tiles and
chunks that are not full, and the smallest and largest dimension they take.

Messages have Frobenius norm 1.  Up to four contractions of up to 64 terms,
each term within 2^-23 of its product of complex64 operands: 4 x 64 x 2^-23 =
3.1e-5 bounds the relative error of a message, 3.5e-5 is asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

DIMS = [(64, 64), (33, 40), (64, 3, 33), (2, 64, 48), (31, 37, 5), (5, 60, 7, 3), (32, 41, 6), (33, 33, 9), (8, 64, 34, 2), (63, 2, 2, 2),
        (3, 3, 64, 11)]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_wide_site_matches_oracle(dims, prec):
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
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        tb.BeliefPropagation(st)
        assert max(float(np.max(np.abs(st.get_message(m) - F[m]))) for m in range(2 * ne)) <= 3.5e-5


# Even extents that end inside a group of four columns, tiles that are not full
FORMS = [(50, 3), (34, 7, 3), (42, 38, 35), (6, 9, 34, 2)]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("dims", FORMS, ids=["x".join(map(str, d)) for d in FORMS])
def test_memory_forms_match_oracle(dims, prec):
    test_wide_site_matches_oracle(dims, prec)
