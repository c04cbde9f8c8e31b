"""Loops and single sweeps on one job, reduced precision: the condition after a
loop is the one the loop returned (it runs the loop's kernels), other messages
are judged by single sweeps, and a program that changes between the two builds
each plan once (the first again where the second needs a larger scratch)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")
import bp_numpy as bn  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DIMS = (16, 12, 9, 20)
EDGES = [(0, k + 1) for k in range(4)]


def state():
    rng = np.random.default_rng(7)
    gauss = lambda sh: rng.normal(size=sh) + 1j * rng.normal(size=sh)
    V = [gauss([DIMS[m] for m in bn.bonds_of(EDGES, s)] + [2]) for s in bn.sites_of(EDGES)]
    return V, [np.eye(DIMS[m % 4]) / np.sqrt(DIMS[m % 4]) for m in range(8)]


@pytest.mark.parametrize("prec", [tb.MIXED, tb.C64], ids=["mixed", "c64"])
@pytest.mark.parametrize("sweeps", [1, 3, 50])
def test_condition_after_a_loop_is_the_loops(prec, sweeps):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    V, E = state()
    with tb.State(EDGES, prec) as st:
        st.set_state(V, E)
        first = tb.BeliefPropagationCondition(st)
        _, cond = tb.BeliefPropagationLoop(st, 1e-300, sweeps)
        assert tb.BeliefPropagationCondition(st) == cond
        st.set_state(V, E)  # messages of no loop
        assert tb.BeliefPropagationCondition(st) == first


SCRIPT = """
import sys
sys.path[:0] = [{root!r}, {oracle!r}, {tests!r}]
import tnbp_b200 as tb
from test_gpu_sweep_plans import EDGES, state
V, E = state()
with tb.State(EDGES, tb.MIXED) as st:
    st.set_state(V, E)
    for _ in range(6):
        tb.BeliefPropagationLoop(st, 1e-300, 3)
        tb.BeliefPropagationCondition(st)
        tb.BeliefPropagation(st)
        tb.BeliefPropagationCondition(st)
"""


@pytest.mark.parametrize("wave_mb", ["0", "1"])  # one wave, several
def test_changing_between_loops_and_single_sweeps_keeps_both_plans(wave_mb):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    code = SCRIPT.format(root=ROOT, oracle=os.path.join(ROOT, "oracle"), tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, TNBP_TRACE="1", TNBP_WAVE_MB=wave_mb), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    builds = [int(l.split()[1]) for l in r.stderr.splitlines() if l.split()[:1] == ["sweep.build_plan"]]
    # one more at most: the second plan may need a larger scratch than the first was built on
    assert len(builds) == 1 and builds[0] <= 3, r.stderr[-2000:]
