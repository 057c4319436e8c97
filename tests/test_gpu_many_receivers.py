"""Receivers by the thousand in the two-kernel step: on either side of the number up to which the velocity kernel
samples them, against the oracle, and at a cost that stays near the step's own."""
import time

import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch, Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _spread(m, n, stress):
    rng = np.random.default_rng(n)
    rec = np.stack([rng.integers(1, m.nx, n), rng.integers(1, m.ny, n), rng.integers(1, m.nz, n), rng.integers(0, 3, n)], 1)
    if stress:
        rec[n // 2] = (0, 3, 1, F.F_SXY)
    m.receivers = rec.astype(np.int32)


@pytest.mark.parametrize("precision", [F.PREC_F32, F.PREC_F32_KAHAN, F.PREC_F64])
@pytest.mark.parametrize("n,stress", [(255, True), (257, True), (8192, False), (8193, False), (40000, True)])
def test_against_the_oracle(cuda_device, precision, n, stress):
    m = I.random_small(F.MODEL_ORTHO, 37, 26, 19, nt=20, seed=3, damping=F.DAMP_SEPARABLE)
    _spread(m, n, stress)
    ref = O.run(m, 20, precision)
    with Solver.from_model(m, precision=precision) as s:
        for k in (3, 8, 9):
            s.run(k)
        np.testing.assert_array_equal(s.seismograms(), ref.traces)


@pytest.mark.parametrize("n", [8192, 8193])
def test_in_a_batch(cuda_device, n):
    m = I.random_small(F.MODEL_ISO, 37, 26, 19, nt=20, seed=3)
    _spread(m, n, False)
    ref = O.run(m, 20)
    with Batch([(m, [(m.sources, m.source_coef)] * 2)]) as b:
        for k in (3, 17):
            b.run(k)
        for r in range(2):
            np.testing.assert_array_equal(b.seismograms(0, r), ref.traces)


def test_two_full_planes_cost_less_than_two_steps(cuda_device):
    n, nz, nt = 420, 110, 200
    small = I.random_small(F.MODEL_ISO, n, n, 8, nt=nt, seed=2)
    m = I.Model(**{**small.__dict__, "nz": nz, "materials": {}, "damping_arrays": dict(small.damping_arrays)})
    for q in (F.M_C11, F.M_C12):
        m.materials[q] = np.ones((nz, n, n), np.float32)
    m.damping_arrays[F.D_WZ] = np.ones(nz + 1, np.float32)
    m.set_moment_tensor([1, 1, 1, 0, 0, 0], n // 2, n // 2, 2, stencil=0)
    times = []
    for planes in ((), (1, nz - 1)):
        m.receivers = np.array([(n // 2, n // 2, 1, 0)] + [(i, j, k, 2) for k in planes for j in range(1, n) for i in range(1, n)], np.int32)
        with Solver.from_model(m) as s:
            s.run(32)
            best = 1e9
            for _ in range(3):
                t0 = time.perf_counter()
                s.run(48)
                best = min(best, time.perf_counter() - t0)
                s.reset()
            times.append(best / 48)
    assert times[1] < 3 * times[0], times  # 1.7 times; 4 with one CTA for all receivers
