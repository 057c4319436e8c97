"""What the autotuner returns makes a handle or a batch of the same setting."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu


def _step_us(s):
    s.run(64)
    best = 1e9
    for _ in range(5):
        s.reset()
        best = min(best, s.run(256))
    return best / 256 * 1e3


@pytest.mark.parametrize("n", [40, 50, 80])  # chunks of one and of two planes by the rule
def test_solver(cuda_device, n):
    """With the four planes that 4 stood for, 50^3 took 1.3 times the tuned setting's time."""
    m = I.random_small(F.MODEL_ISO, n, n, n, nt=400, seed=1)
    with Solver.from_model(m) as s:
        k = s.autotune(30)
        ty, pf = s.tile(), s.l2_prefetch()
        tuned = _step_us(s)
        ref = s.seismograms()
    with Solver.from_model(m, kchunk=k) as s:
        s.set_tile(ty)
        s.set_l2_prefetch(pf)
        again = _step_us(s)
        np.testing.assert_array_equal(s.seismograms(), ref)
    with Solver.from_model(m) as s:
        default = _step_us(s)
    assert again < 1.15 * tuned and tuned < 1.15 * default, (k, ty, pf, tuned, again, default)


def _problems():
    probs = []
    for n, model in ((40, F.MODEL_ISO), (40, F.MODEL_ISO), (52, F.MODEL_ORTHO)):
        m = I.random_small(model, n, n, n, nt=400, seed=n)
        probs.append((m, [(m.sources, m.source_coef)] * (2 if model == F.MODEL_ORTHO else 1)))
    return probs


def test_batch(cuda_device):
    with Batch(_problems()) as b:
        assert (b.tile(), b.l2_prefetch(), b.launch()) == (4, 0, 0)
        b.run(64)
        default = _step_us(b)
        b.set_l2_prefetch(b.l2_prefetch())  # the defaults can be put back
        b.set_launch(b.launch())
        same = _step_us(b)
        k = b.autotune(20)
        setting = b.tile(), b.l2_prefetch(), b.launch()
        tuned = _step_us(b)
        ref = [b.seismograms(p, 0) for p in range(3)]
    with Batch(_problems(), kchunk=k) as b:
        b.set_tile(setting[0])
        b.set_l2_prefetch(setting[1])
        b.set_launch(setting[2])
        again = _step_us(b)
        for p in range(3):
            np.testing.assert_array_equal(b.seismograms(p, 0), ref[p])
    assert same < 1.15 * default and again < 1.15 * tuned and tuned < 1.15 * default, (k, setting, default, same, tuned, again)
