"""The pair-of-legs kernels on lattices whose bonds all differ: their
persistent CTAs walk through several tasks each, of other dimensions, memory
forms and sizes (small ones after large ones, both plane counts), and every
message agrees with the numpy oracle.

A message has Frobenius norm 1; four stages leave a few 2^-23 (see the wide
kernels' test), 1e-6 is asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

SIZES = [1, 2, 3, 4, 5, 6, 7, 9, 12, 16, 17, 20, 25, 32]
WEIGHTS = {"small": [2, 6, 8, 7, 5, 4, 4, 4, 3, 2, 1, 1, 0, 1], "even": [0, 9, 0, 9, 0, 6, 0, 0, 4, 4, 0, 2, 0, 1]}


def pair_tasks(edges, dims):
    """(planes, tiles) of each pair task, in site order."""
    out = []
    for s in bn.sites_of(edges):
        D = [dims[m] for m in bn.bonds_of(edges, s)]
        if len(D) != 4 or max(D) <= 8:
            continue
        for x in (0, 2):
            planes = 8 if max(D[x], D[x + 1]) <= 16 else 4
            n_outer = 2 * int(np.prod(D)) // (D[x] * D[x + 1])
            out.append((planes, -(-n_outer // planes)))
    return out


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("kind", list(WEIGHTS))
def test_ragged_lattice_matches_oracle(kind, prec):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    rng = np.random.default_rng(len(kind))
    edges = tb.bond_square_lattice(18, 18)
    w = np.array(WEIGHTS[kind], float)
    dims = [int(d) for d in rng.choice(SIZES, size=len(edges), p=w / w.sum())]
    tasks = pair_tasks(edges, dims)
    for planes in (4, 8):  # a CTA's equal share of the tiles holds several of most tasks
        tiles = [t for p, t in tasks if p == planes]
        share = -(-sum(t for _, t in tasks) // 148)
        assert len(tiles) > 50 and np.mean([2 * t < share for t in tiles]) > 0.4
        assert any(a > 4 * b for a, b in zip(tiles, tiles[1:]))
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = []
    for s in bn.sites_of(edges):
        v = gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2])
        V.append(v / np.linalg.norm(v))
    E = []
    for m in range(2 * len(edges)):
        A = gauss((dims[m % len(edges)],) * 2)
        M = A @ A.conj().T
        E.append(M / np.linalg.norm(M))
    F = bn.bp_sweep(edges, V, E)
    with tb.State(edges, prec) as st:
        st.set_state(V, E)
        for _ in range(2):  # twice from the same messages: nothing is left behind
            for m, e in enumerate(E):
                st.set_message(m, e)
            tb.BeliefPropagationLoop(st, 1e-300, 1)
            assert max(float(np.linalg.norm(a - b)) for a, b in zip(st.get_E(), F)) <= 1e-6
