"""The pair-of-legs kernels of the reduced-precision sweeps (tc_pair.cuh)
against the numpy oracle: a degree-4 site with the bond dimensions at which
their tiles change (planes per tile, half ranges of 4, 8, 12 and 16 columns,
unequal dimensions in a pair, a last tile that is not full, odd dimensions
and outer strides, dimension 1, and 33, which is left to the other kernels).

Messages have Frobenius norm 1.  Four contractions of up to 32 terms, each
term within 2^-23 of its product of complex64 operands: 4 x 32 x 2^-23 =
1.5e-5 bounds the relative error of a message, 2e-5 is asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

DIMS = [(32, 32, 32, 32), (16, 16, 16, 16), (8, 8, 8, 8), (31, 17, 8, 5), (24, 20, 12, 9), (5, 32, 6, 4), (7, 7, 11, 13), (1, 30, 25, 3),
        (2, 3, 32, 32), (10, 18, 26, 4), (33, 8, 6, 5)]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_degree_four_site_matches_oracle(dims, prec):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    rng = np.random.default_rng(sum(dims))
    edges = [(0, k + 1) for k in range(4)]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = []
    for m in range(8):
        A = gauss((dims[m % 4],) * 2)
        M = A @ A.conj().T
        E.append(M / np.linalg.norm(M))
    F = bn.bp_sweep(edges, V, E)
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        for _ in range(2):  # twice from the same messages: nothing is left behind
            for m in range(8):
                st.set_message(m, E[m])
            tb.BeliefPropagationLoop(st, 1e-300, 1)  # its sweeps take pairs of legs
            got = [st.get_message(m) for m in range(8)]
            assert max(float(np.max(np.abs(a - b))) for a, b in zip(got, F)) <= 2e-5


# Where a plane's elements run along memory or consecutive planes do, in
# copies of two elements or (odd extents) of one
FORMS = [(1, 1, 32, 32), (1, 1, 17, 9), (2, 1, 9, 8), (3, 1, 32, 32), (2, 5, 16, 16), (1, 4, 31, 7), (12, 2, 3, 1), (30, 14, 23, 24)]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("dims", FORMS, ids=["x".join(map(str, d)) for d in FORMS])
def test_memory_forms_match_oracle(dims, prec):
    test_degree_four_site_matches_oracle(dims, prec)


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
def test_single_sweeps_do_not_depend_on_the_loop(prec):
    """A sweep between loops gives the bits of a sweep without one."""
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    rng = np.random.default_rng(7)
    dims = (16, 12, 9, 20)
    edges = [(0, k + 1) for k in range(4)]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = [np.eye(dims[m % 4]) / np.sqrt(dims[m % 4]) for m in range(8)]
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        out = []
        for step in (tb.BeliefPropagation, lambda s: tb.BeliefPropagationLoop(s, 1e-300, 1), tb.BeliefPropagation):
            for m in range(8):
                st.set_message(m, E[m])
            step(st)
            out.append([st.get_message(m) for m in range(8)])
        assert all(np.array_equal(a, b) for a, b in zip(out[0], out[2]))
        assert max(float(np.max(np.abs(a - b))) for a, b in zip(out[0], out[1])) <= 2e-5
