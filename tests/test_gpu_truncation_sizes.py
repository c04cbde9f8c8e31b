"""The truncation kernels (k_trunc_roots, k_truncate_edges) against the numpy
oracle at the bond dimensions where their layout changes: 16 lanes per column
pair (rows held as 1, 2, 4 or 5 registers per lane), odd dimensions (one
column idles per round), one and two columns, matrices in shared memory up to
80 and in global memory above, several dimensions in one launch, and messages
far from unit scale.  Kept dimensions exact; truncation errors, kept singular
values and expectation values at the 1e-10 of the other truncation tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

CASES = [((1,), 4, 1.0), ((2,), 1, 1.0), ((3, 15), 4, 1.0), ((16, 17), 16, 1.0), ((31, 32, 33), 16, 1.0), ((63, 2), 40, 1.0),
         ((64, 5), 32, 1.0), ((65, 80), 33, 1.0), ((81, 8), 81, 1.0), ((128, 3), 20, 1.0), ((12, 7, 30), 8, 1e-60), ((24, 9), 12, 1e40)]


@pytest.mark.parametrize("dims,chi,scale", CASES, ids=["x".join(map(str, c[0])) + "-%g" % c[2] for c in CASES])
def test_truncation_matches_oracle(dims, chi, scale):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    rng = np.random.default_rng(sum(dims) + chi)
    sv_min = 1e-8 * min(1.0, scale)
    edges = [(0, k + 1) for k in range(len(dims))]  # a star
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = []
    for m in range(2 * len(edges)):
        D = dims[m % len(edges)]
        A = gauss((D, 2 * D))  # condition number of a few tens
        M = A @ A.conj().T
        E.append(scale * M / np.linalg.norm(M))
    with tb.State(edges, tb.C128) as st:
        st.set_state(V, E)
        got_dims, got_errs = tb.Truncation(st, chi, sv_min)
        s = [np.diag(st.get_message(m)).real for m in range(len(edges))]
        z = tb.Measure(st, [0], [bn.pauli_op("X")])[0]
    Vt, Et, want_dims, want_errs = bn.truncate(edges, V, E, chi, sv_min)
    assert list(got_dims) == [int(d) for d in want_dims]
    assert np.max(np.abs(np.asarray(got_errs) - np.asarray(want_errs))) <= 1e-10
    for m in range(len(edges)):
        assert np.max(np.abs(s[m] - np.diag(Et[m]).real)) <= 1e-10
    assert abs(z - bn.measure_1site(edges, Vt, Et, 0, bn.pauli_op("X"))) <= 1e-10
