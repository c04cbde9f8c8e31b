"""The mixed path's loops sweep sites whose bond dimensions are all at most 8
in complex128: their messages agree with the numpy oracle to FP64 rounding,
on chip (small sites) and level by level, and a site with a larger bond keeps
the reduced-precision kernels.

A message has Frobenius norm 1.  Its elements are sums of at most 8 products
on each of up to 7 legs and of at most 2 x 8^3 in the Gram (64 for the small
ones), so the rounding of FP64 sums of n terms, n 2^-53 of the absolute sum,
stays below 1100 x 1.1e-16 = 1.2e-13 of sums whose cancellation is mild for
positive messages; 1e-12 is asked for.  Complex64 tensors alone put it at 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402


def star(dims, seed):
    rng = np.random.default_rng(seed)
    g = len(dims)
    edges = [(0, k + 1) for k in range(g)]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = []
    for m in range(2 * g):
        A = gauss((dims[m % g],) * 2)
        E.append(A @ A.conj().T / np.linalg.norm(A @ A.conj().T))
    return edges, V, E


def loop_error(dims, prec=tb.MIXED):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    edges, V, E = star(dims, sum(dims))
    F = bn.bp_sweep(edges, V, E)
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        tb.BeliefPropagationLoop(st, 1e-300, 1)
        return max(float(np.linalg.norm(st.get_message(m) - F[m])) for m in range(len(dims)))


@pytest.mark.parametrize("dims", [(8, 8, 8, 8), (8, 5, 7, 8), (6, 6, 6, 6), (4, 4, 4, 4), (8, 8, 8), (3, 2, 5, 4, 2), (1, 8), (7,)],
                         ids=lambda d: "x".join(map(str, d)))
def test_small_sites_are_swept_in_complex128(dims):
    assert loop_error(dims) <= 1e-12


def test_larger_bonds_and_complex64_storage_are_not():
    assert 1e-10 < loop_error((9, 8, 8, 8)) <= 2e-5
    assert 1e-10 < loop_error((8, 8, 8, 8), tb.C64) <= 2e-5
