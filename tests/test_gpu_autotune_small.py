"""The autotuners where the host does not keep up with launches one by one: the pick is not slower than the rule by
size, run as users run it."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu


def _step_us(s, n=640):
    s.run(n)
    best = 1e9
    for _ in range(4):
        s.reset()
        best = min(best, s.run(n))
    return best / n * 1e3


@pytest.mark.parametrize("rounds", range(3))
def test_batch_of_small_chains(cuda_device, rounds):
    """Launched one by one, every setting of these 40 chains takes the host's 200 us a step; the settings differ by a factor of two."""
    probs = []
    for q in range(40):
        m = I.random_small(F.MODEL_ISO, 34, 34, 34, nt=640, seed=q % 4)
        probs.append((m, [(m.sources, m.source_coef)]))
    with Batch(probs) as b:
        default = _step_us(b)
        b.autotune(8)
        setting = b.tile(), b.l2_prefetch(), b.launch()
        assert _step_us(b) < 1.1 * default, setting


@pytest.mark.parametrize("shape", [(24, 24, 24), (40, 40, 32), (64, 48, 40)])
@pytest.mark.parametrize("nsteps", [1, 3, 20])
def test_solver_on_small_grids(cuda_device, shape, nsteps):
    m = I.random_small(F.MODEL_ORTHO, *shape, nt=640, seed=5, damping=F.DAMP_SEPARABLE)
    with Solver.from_model(m) as s:
        default = _step_us(s)
        ref = s.seismograms()
        s.reset()
        k = s.autotune(nsteps)
        assert s.step() == 0
        tuned = _step_us(s)
        np.testing.assert_array_equal(s.seismograms(), ref)
    assert tuned < 1.1 * default, (k, tuned, default)
