"""Batch chains: sources and receivers that the step's own kernels take and those that need the separate
ones, per right-hand side, and runs split at odd steps, against the oracle, bit for bit."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch
from oracle import oracle as O

pytestmark = pytest.mark.gpu

COMP = (F.F_SXX, F.F_SZZ, F.F_SXY, F.F_SXZ, F.F_SYZ)


def _problem(model, shape, nt, nrhs, seed, outside, stress_rec, **kw):
    """outside: one right-hand side has a source on the face that the stress update leaves out."""
    m = I.random_small(model, *shape, nt=nt, seed=seed, **kw)
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    rhs = []
    for r in range(nrhs):
        n = (7, 30, 0, 1)[r % 4]                             # in the parameters, in device memory, none, one
        ent = [(COMP[rng.integers(5)], rng.integers(nx), rng.integers(ny), rng.integers(nz)) for _ in range(n)]
        ent += [(F.F_SXZ, 5 + r, 4, 1), (F.F_SXX, 3, 3 + r, 0)] if n else []
        if outside and r == nrhs - 1:
            ent.append((F.F_SXY, nx, 4, 2))
        rhs.append((np.array(ent, np.int32).reshape(-1, 4), rng.normal(size=len(ent))))
    rec = [(i, j, k, c) for i, j in ((1, 1), (2, 1), (nx - 1, ny - 1)) for k in (1, 2, nz - 1) for c in range(3)]
    if stress_rec:
        rec.append((0, 3, 1, F.F_SXY))
    m.receivers = np.array(rec, np.int32)
    return m, rhs


@pytest.mark.parametrize("own", [0, 1])
@pytest.mark.parametrize("outside,stress_rec", [(False, False), (True, False), (False, True), (True, True)])
def test_chains(cuda_device, own, outside, stress_rec):
    nt = 150
    probs = [_problem(F.MODEL_ISO, (34, 21, 12), nt, 1, 3, outside, stress_rec),
             _problem(F.MODEL_ORTHO, (23, 33, 9), nt, 4, 4, outside, stress_rec, damping=F.DAMP_W3D),
             _problem(F.MODEL_ORTHO, (33, 18, 8), nt, 1, 5, False, stress_rec, damping=F.DAMP_SEPARABLE),
             _problem(F.MODEL_ISO, (31, 20, 7), nt, 2, 6, outside, False, src_order=F.SRC_AFTER_BC1),
             _problem(F.MODEL_ORTHO, (90, 80, 60), nt, 1, 7, outside, stress_rec, damping=F.DAMP_SEPARABLE)]  # two cells per thread
    with Batch(probs) as b:
        b.set_launch(own)
        for n in (1, 2, 67, 66, 14):  # a step; two; one and a graph from step 3 on; graph and two; rest
            b.run(n)
        for p, (m, rhs) in enumerate(probs):
            for r, (ent, coef) in enumerate(rhs):
                m.sources, m.source_coef = ent, coef
                ref = O.run(m, nt)
                np.testing.assert_array_equal(b.seismograms(p, r), ref.traces, err_msg=f"problem {p} rhs {r}")
                for q in F.STATE:
                    np.testing.assert_array_equal(b.field(p, r, q), ref.f[q], err_msg=f"problem {p} rhs {r} {F.STATE_NAMES[q]}")


@pytest.mark.parametrize("model,damping", [(F.MODEL_ISO, None), (F.MODEL_ORTHO, F.DAMP_SEPARABLE), (F.MODEL_ORTHO, F.DAMP_W3D)])
@pytest.mark.parametrize("outside,stress_rec", [(False, False), (True, True)])
def test_shared_launches(cuda_device, model, damping, outside, stress_rec):
    """A model large enough for its right-hand sides to share launches."""
    nt, shape = 9, (139, 137, 133)
    assert np.prod(shape) >= 2.5e6
    m, rhs = _problem(model, shape, nt, 4, 8, outside, stress_rec, **({} if damping is None else {"damping": damping}))
    with Batch([(m, rhs)]) as b:
        for n in (3, 6):
            b.run(n)
        for r, (ent, coef) in enumerate(rhs):
            m.sources, m.source_coef = ent, coef
            ref = O.run(m, nt)
            np.testing.assert_array_equal(b.seismograms(0, r), ref.traces, err_msg=f"rhs {r}")
            for q in F.STATE:
                np.testing.assert_array_equal(b.field(0, r, q), ref.f[q], err_msg=f"rhs {r} {F.STATE_NAMES[q]}")


@pytest.mark.parametrize("own", [0, 1])
def test_many_tiny_problems(cuda_device, own):
    """Problems small and many enough for one launch over all of a scheme's, among others that are not."""
    nt = 80
    rng = np.random.default_rng(12)
    probs = []
    for q in range(46):
        shape = tuple(int(v) for v in rng.integers(7, 35, 2)) + (int(rng.integers(4, 14)),)
        model, kw = ((F.MODEL_ISO, {}), (F.MODEL_ORTHO, {"damping": F.DAMP_SEPARABLE}))[q % 2] if q < 44 else (F.MODEL_ORTHO, {"damping": F.DAMP_W3D})
        if q % 6 == 0:
            kw = {**kw, "src_order": F.SRC_AFTER_BC1}
        # 0: seven entries and two near the surface; some with a source or a receiver for the separate kernels
        probs.append(_problem(model, shape, nt, 1 if q % 12 else 2, 20 + q, q in (3, 4), q in (4, 7), **kw))
    with Batch(probs) as b:
        b.set_launch(own)
        for n in (1, 2, 67, 10):
            b.run(n)
        for p, (m, rhs) in enumerate(probs):
            for r, (ent, coef) in enumerate(rhs):
                m.sources, m.source_coef = ent, coef
                ref = O.run(m, nt)
                np.testing.assert_array_equal(b.seismograms(p, r), ref.traces, err_msg=f"problem {p} rhs {r}")
                for q in F.STATE:
                    np.testing.assert_array_equal(b.field(p, r, q), ref.f[q], err_msg=f"problem {p} rhs {r} {F.STATE_NAMES[q]}")
