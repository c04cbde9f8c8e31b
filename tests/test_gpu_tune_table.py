"""The wave budgets of the tuning table belong to one schedule and one version
of the kernels: an entry of an earlier table, or of the loops' plans, does not
change how single sweeps are split (seen in their number of launches), and an
entry of their own does."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
sys.path.insert(0, {root!r})
import numpy as np, tnbp_b200 as tb
edges = tb.bond_square_lattice(3, 3)
rng = np.random.default_rng(3)
sites = sorted({{v for e in edges for v in e}})
with tb.State(edges, tb.MIXED) as st:
    for r in (4, 4):
        ops = [rng.normal(size=[r] * sum(s in e for e in edges) + [2, 2]) + 0j for s in sites]
        tb.AbsorbTPO(st, tb.TPOLayer.from_ops(edges, ops))
    out = []
    for step in (tb.BeliefPropagation, lambda s: tb.BeliefPropagationLoop(s, 1e-300, 1)):
        n = tb.kernel_launches()
        step(st)
        out.append(tb.kernel_launches() - n)
print(*out)
"""


def launches(tmp_path, name, keys):
    import torch

    p = torch.cuda.get_device_properties(0)
    d = tmp_path / name
    d.mkdir()
    dev = "".join(c if c.isalnum() else "_" for c in p.name)
    with open(d / f"waves_{dev}_{p.multi_processor_count}sm.tsv", "w") as f:
        for k in keys:
            f.write(f"{k}\t1\t1.0\t2.0\n")
    env = dict(os.environ, TNBP_TUNE_DIR=str(d))
    env.pop("TNBP_WAVE_MB", None)
    env.pop("TNBP_AUTOTUNE", None)
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [int(x) for x in r.stdout.split()]


def test_budgets_are_kept_per_schedule_and_kernel_version(tmp_path):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    key = "mixed_D16_g4_n16"
    single, loop = launches(tmp_path, "none", [])
    assert launches(tmp_path, "earlier", [key]) == [single, loop]
    s, l = launches(tmp_path, "loops", [key + "_loop_k2"])
    assert s == single and l > loop
    s, l = launches(tmp_path, "single", [key + "_single_k2"])
    assert s > single and l == loop
