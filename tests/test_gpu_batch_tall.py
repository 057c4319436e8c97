"""Batches of a grid with more planes than 65535 chunks of the size asked for, and with more rows than 65535 CTAs have."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Batch

pytestmark = pytest.mark.gpu


def test_more_planes_than_chunks(cuda_device):
    nz, nt = 4 * 65535 + 61, 40
    small = I.random_small(F.MODEL_ISO, 9, 7, 12, nt=nt, seed=6)
    m = I.Model(**{**small.__dict__, "nz": nz, "materials": {}, "damping_arrays": dict(small.damping_arrays)})
    for q, a in small.materials.items():
        m.materials[q] = np.full((nz, 7, 9), a[0, 0, 0], np.float32)
    m.damping_arrays[F.D_WZ] = np.ones(nz + 1, np.float32)
    m.set_moment_tensor([1, 1, 1, 0.2, 0, 0], 3, 2, nz - 20, stencil=0)
    m.receivers = np.array([(4, 3, k, c) for k in (nz - 30, nz - 12, nz - 1) for c in range(3)], np.int32)
    traces = []
    for kchunk in (0, 4, 32):
        with Batch([(m, [(m.sources, m.source_coef)])], kchunk=kchunk) as b:
            b.run(nt)
            traces.append(b.seismograms(0, 0))
    assert np.abs(traces[0]).max() > 0
    np.testing.assert_array_equal(traces[1], traces[0])
    np.testing.assert_array_equal(traces[2], traces[0])


def test_more_rows_than_ctas(cuda_device):
    """The wave does not reach a row that only the longer grid has."""
    nt, traces = 30, []
    for ny in (60, 16 * 65535 + 61):
        m = I.random_small(F.MODEL_ISO, 9, 11, 6, nt=nt, seed=6)
        base = dict(m.materials)
        m = I.Model(**{**m.__dict__, "ny": ny, "materials": {}, "damping_arrays": dict(m.damping_arrays)})
        for q, a in base.items():
            m.materials[q] = np.full((6, ny, 9), a[0, 0, 0], np.float32)
        m.damping_arrays[F.D_WY] = np.ones(ny + 1, np.float32)
        m.set_moment_tensor([1, 1, 1, 0.2, 0, 0], 3, 5, 2, stencil=0)
        m.receivers = np.array([(4, j, 2, c) for j in (3, 9, 15) for c in range(3)], np.int32)
        with Batch([(m, [(m.sources, m.source_coef)])]) as b:
            b.run(nt)
            traces.append(b.seismograms(0, 0))
    assert np.abs(traces[0]).max() > 0
    np.testing.assert_array_equal(traces[1], traces[0])
