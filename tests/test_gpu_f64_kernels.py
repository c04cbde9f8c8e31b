"""The FP64 tensor-pipe kernels (k_leg_apply_f64, k_gram_f64) against the numpy
oracle at the sizes where their tiles end: star graphs whose centre has bond
dimensions around the 8-, 16-, 32- and 64-wide edges of the tiles, with leg
strides of 1, odd, just below and above 32 (whole-block tiles end there) and
above 64, and the largest supported dimension, 128.

TNBP_SITE_SWEEP=0 sends every site through these kernels; the switch is read
once per process, so one child process runs every shape.  One sweep and the
one- and two-site environments each; messages are normalized and the values
are ratios, both compared at the 1e-12 of the complex128 sweep tests.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SHAPES = [(1, 2, 3), (2, 5, 3), (4, 4, 4, 4), (7, 3, 9), (9, 16, 8), (5, 13, 17), (31, 4, 5), (32, 3, 12), (33, 2, 31), (3, 11, 33),
          (17, 2, 3, 24), (64, 7), (65, 6), (5, 64, 2), (128, 3, 2), (3, 128), (2, 2, 2, 2, 2, 3)]

SCRIPT = r"""
import json, sys
import numpy as np
sys.path[:0] = [{root!r}, {oracle!r}]
import tnbp_b200 as tb, bp_numpy as bn
out = []
for dims in {shapes!r}:
    rng = np.random.default_rng(sum(dims))
    edges = [(0, k + 1) for k in range(len(dims))]
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([dims[m] for m in bn.bonds_of(edges, s)] + [2]) for s in bn.sites_of(edges)]
    E = []
    for m in range(2 * len(edges)):
        A = gauss((dims[m % len(edges)],) * 2)
        M = A @ A.conj().T
        E.append(M / np.linalg.norm(M))
    with tb.State(edges, tb.C128) as st:
        st.set_state(V, E)
        one = tb.Measure(st, [0], [bn.pauli_op("Y")])[0] - bn.measure_1site(edges, V, E, 0, bn.pauli_op("Y"))
        two = max(abs(a - bn.measure_2site(edges, V, E, p, bn.pauli_two("X", "Y")))
                  for p, a in zip(edges, tb.Measure(st, edges, [bn.pauli_two("X", "Y")] * len(edges))))
        tb.BeliefPropagation(st)
        F = bn.bp_sweep(edges, V, E)
        msg = max(float(np.max(np.abs(st.get_message(m) - F[m]))) for m in range(2 * len(edges)))
    out.append([msg, float(abs(one)), float(two)])
print("RESULT" + json.dumps(out))
"""


@pytest.fixture(scope="module")
def errors():
    env = dict(os.environ, TNBP_SITE_SWEEP="0")
    code = SCRIPT.format(root=ROOT, oracle=os.path.join(ROOT, "oracle"), shapes=SHAPES)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.split("RESULT")[-1])


@pytest.mark.parametrize("i", range(len(SHAPES)), ids=["x".join(map(str, s)) for s in SHAPES])
def test_star_matches_oracle(errors, i):
    assert max(errors[i]) <= 1e-12, errors[i]
