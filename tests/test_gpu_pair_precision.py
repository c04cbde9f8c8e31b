"""Precision of the pair-of-legs kernels (tc_pair.cuh): the messages that a
loop's sweep sends from a degree-4 site are no further from the 64-bit ones
than those of a single sweep, whose legs and Grams are separate kernels, over
twelve seeds (three at D = 32), with and without decay along the bonds.

The tensors are complex64 values and the messages complex128, so all of the
error is the sweep's own.  Beside it the error that plain TF32 operands would
leave (no lo parts) is computed and has to be far larger, so that a lost split
cannot pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

EDGES = [(0, k + 1) for k in range(4)]
DIMS = [(32, 32, 32, 32), (16, 16, 16, 16), (12, 12, 12, 12), (24, 20, 12, 9), (31, 17, 8, 5), (1, 30, 25, 3), (2, 3, 32, 32)]


def make(dims, kind, seed):
    rng = np.random.default_rng([seed, sum(dims)])
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = []
    for s in bn.sites_of(EDGES):
        sh = [dims[m] for m in bn.bonds_of(EDGES, s)] + [2]
        v = gauss(sh)
        if kind == "decay":
            for k in range(len(sh) - 1):
                v = v * (0.8 ** np.arange(sh[k])).reshape([-1 if j == k else 1 for j in range(len(sh))])
        V.append((v / np.linalg.norm(v)).astype(np.complex64).astype(np.complex128))
    E = []
    for m in range(8):
        D = dims[m % 4]
        A = gauss((D, D))
        M = A @ A.conj().T
        if kind == "decay":
            M = M * 0.05 / D + np.diag(0.7 ** np.arange(D))
        E.append(M / np.linalg.norm(M))
    return V, E


def tf32(a):
    """Rounded to 11 significant bits."""
    def part(x):
        bits = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
        return ((bits + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32).astype(np.float64)
    return part(a.real) + 1j * part(a.imag)


def plain_tf32(V, E, k):
    """Message k with TF32 operands everywhere."""
    t = tf32(V)
    for j in range(4):
        if j != k:
            t = tf32(np.moveaxis(np.tensordot(t, tf32(E[j + 4]), axes=([j], [0])), -1, j))
    rest = [i for i in range(5) if i != k]
    return bn.normalize(np.tensordot(t, tf32(V).conj(), axes=(rest, rest)))[0]


@pytest.mark.parametrize("kind", ["gauss", "decay"])
@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_loop_sweeps_are_as_exact_as_single_ones(dims, kind):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    seeds = 3 if min(dims) == 32 else 12
    legs = [k for k in range(4) if dims[k] > 1]
    err = {"single": [], "loop": [], "tf32": []}
    for seed in range(seeds):
        V, E = make(dims, kind, seed)
        F = bn.bp_sweep(EDGES, V, E)
        with tb.State(EDGES, tb.MIXED) as st:
            for name, step in (("single", tb.BeliefPropagation), ("loop", lambda s: tb.BeliefPropagationLoop(s, 1e-300, 1))):
                st.set_state(V, E)
                step(st)
                err[name] += [np.linalg.norm(st.get_message(k) - F[k]) for k in legs]
        if seed == 0:
            err["tf32"] += [np.linalg.norm(plain_tf32(V[0], E, k) - F[k]) for k in legs]
    rms = {k: float(np.sqrt(np.mean(np.square(v)))) for k, v in err.items()}
    assert rms["loop"] <= rms["single"], rms
    assert rms["tf32"] >= 10 * rms["single"], rms
