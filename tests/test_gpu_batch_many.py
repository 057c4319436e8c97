"""Tiny problems in shared launches around the numbers and sizes at which they share them, with sources and receivers
that those launches take and that they do not, against the oracle, bit for bit."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _problem(model, shape, nt, seed, outside, stress, **kw):
    m = I.random_small(model, *shape, nt=nt, seed=seed, **kw)
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    ent = [(c, *rng.integers(1, (nx, ny, nz))) for c in (F.F_SXX, F.F_SXZ)] + ([(F.F_SYZ, 4, ny, 2)] if outside else [])
    m.sources, m.source_coef = np.array(ent, np.int32), rng.normal(size=len(ent))
    m.receivers = np.array([(2, 3, 1, F.F_VX), (nx - 1, ny - 1, nz - 1, F.F_VZ)] + ([(0, 3, 1, F.F_SZZ)] * 2 if stress else []), np.int32)
    return m, [(m.sources, m.source_coef)]


@pytest.mark.parametrize("model,kw", [(F.MODEL_ISO, {}), (F.MODEL_ORTHO, {"damping": F.DAMP_SEPARABLE}), (F.MODEL_ORTHO, {"damping": F.DAMP_W3D})])
@pytest.mark.parametrize("small,large", [(11, 0), (12, 0), (12, 19), (12, 20), (0, 32), (3, 31)])
def test_many(cuda_device, model, kw, small, large):
    nt = 21
    probs = [_problem(model, (9 + q % 5, 11, 5 + q % 3), nt, q, q % 4 == 1, q % 4 == 2, **kw) for q in range(small)]
    probs += [_problem(model, (33, 27, 24), nt, 50 + q, q % 8 == 1, q % 8 == 2, **kw) for q in range(large)]
    assert not large or 2e4 <= 33 * 27 * 24 < 2.8e4
    with Batch(probs) as b:
        for n in (1, 8, 11, 1):
            b.run(n)
        for p, (m, _) in enumerate(probs):
            ref = O.run(m, nt)
            np.testing.assert_array_equal(b.seismograms(p, 0), ref.traces, err_msg=f"problem {p}")
            np.testing.assert_array_equal(b.field(p, 0, F.F_VX), ref.f[F.F_VX], err_msg=f"problem {p}")
