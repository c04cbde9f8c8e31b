"""An AbsorbTPO that is refused (a site tensor of 2^31 elements or more) leaves
the job as it was: bond dimensions, tensors and messages, and the mixed path's
complex64 copy, so that the sweep after it gives the bits of a job that never
saw the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

tb = pytest.importorskip("tnbp_b200")

EDGES = [(0, k + 1) for k in range(4)]


def layer(ranks, seed):
    rng = np.random.default_rng(seed)
    gauss = lambda sh: (rng.normal(size=sh) + 1j * rng.normal(size=sh)) / 2
    return tb.TPOLayer.from_ops(EDGES, [gauss(list(ranks) + [2, 2])] + [gauss([r, 2, 2]) for r in ranks])


@pytest.mark.parametrize("prec", [tb.C128, tb.MIXED, tb.C64], ids=["c128", "mixed", "c64"])
def test_refused_absorption_changes_nothing(prec):
    if not tb.device_available():
        pytest.fail("no CUDA device: the GPU tests need a B200")
    first, huge = layer((16, 16, 12, 10), 1), layer((16, 16, 22, 26), 2)  # 256 x 256 x 264 x 260 x 2 elements
    out = []
    for refuse in (False, True):
        with tb.State(EDGES, prec) as st:
            tb.AbsorbTPO(st, first)
            tb.BeliefPropagation(st)
            if refuse:
                before = (st.get_V(), st.get_E())
                with pytest.raises(tb.TnbpError) as e:
                    tb.AbsorbTPO(st, huge)
                assert e.value.code == tb.EUNSUPPORTED
                for a, b in zip(before, (st.get_V(), st.get_E())):
                    assert all(np.array_equal(x, y) for x, y in zip(a, b))
            cond = tb.BeliefPropagationCondition(st)
            tb.BeliefPropagation(st)
            out.append((cond, st.get_V(), st.get_E()))
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
