"""The two-kernel step at its default launch shape (one plane per chunk on small grids): sources and
receivers on the planes and columns that chunks and tables share, against the oracle, bit for bit."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(m, nt, **kw):
    ref = O.run(m, nt, **({"precision": kw["precision"]} if "precision" in kw else {}))
    with Solver.from_model(m, **kw) as s:
        s.run(nt)
        np.testing.assert_array_equal(s.seismograms(), ref.traces)
        for q in F.STATE:
            np.testing.assert_array_equal(s.field(q, ref.f[q].dtype), ref.f[q], err_msg=F.STATE_NAMES[q])


@pytest.mark.parametrize("model", [F.MODEL_ISO, F.MODEL_ORTHO, F.MODEL_ISO_HET])
@pytest.mark.parametrize("order", [F.SRC_BEFORE_BC1, F.SRC_AFTER_BC1])
@pytest.mark.parametrize("planes", [(0, 2, 3), (0, 1, 2, 3)])  # without and with shear entries on plane 1
@pytest.mark.parametrize("nsrc", [7, 30])                      # in the kernel's parameters, in device memory
def test_sources_on_the_surface_planes(cuda_device, model, order, planes, nsrc):
    m = I.random_small(model, 37, 33, 9, nt=12, seed=4, src_order=order)
    rng = np.random.default_rng(nsrc)
    ent = [(c, i, j, k) for k in planes for c in (F.F_SXX, F.F_SZZ, F.F_SXY, F.F_SXZ, F.F_SYZ) for i, j in ((0, 5), (9, 0), (31, 32))]
    ent = [ent[q] for q in rng.permutation(len(ent))[:nsrc]]
    m.sources = np.array(ent, np.int32)
    m.source_coef = rng.normal(size=nsrc)
    _check(m, 12)


@pytest.mark.parametrize("nx,ny,nz", [(34, 20, 40), (65, 9, 12)])
def test_receivers_down_a_column_and_repeated(cuda_device, nx, ny, nz):
    m = I.random_small(F.MODEL_ORTHO, nx, ny, nz, nt=20, seed=6)
    rec = [(i, j, k, c) for i, j in ((1, 1), (2, 1), (31, 3), (32, 3), (33, 3), (nx - 1, ny - 1)) for k in range(1, nz, 3) for c in range(3)]
    rec += rec[5:9] + [(2, 1, nz - 1, 2), (2, 1, 1, 0)]          # several rows of one cell and component
    rec = [rec[q] for q in np.random.default_rng(1).permutation(len(rec))]
    m.receivers = np.array(rec, np.int32)
    _check(m, 20)


def test_receivers_beyond_the_table(cuda_device):
    """A spread whose plane offsets would pass the table's limit is sampled by k_record, as stress
    receivers are."""
    n, nz, nt = 420, 110, 6
    m = I.random_small(F.MODEL_ISO, n, n, 8, nt=nt, seed=2)
    base = {q: a[:, :4, :4] for q, a in m.materials.items()}
    m = I.Model(**{**m.__dict__, "nx": n, "ny": n, "nz": nz, "materials": {}, "damping_arrays": dict(m.damping_arrays)})
    for q, a in base.items():
        m.materials[q] = np.full((nz, n, n), a[0, 0, 0], np.float32)
    m.damping_arrays[F.D_WZ] = np.ones(nz + 1, np.float32)
    at = range(1, n, 1)
    m.receivers = np.array([(i, j, k, F.F_VZ) for k in (1, nz - 1) for j in at for i in at], np.int32)
    assert (n - 1) ** 2 * nz > 1 << 24
    m.set_moment_tensor([1, 1, 1, 0, 0, 0], n // 2, n // 2, 2, stencil=0)
    with Solver.from_model(m) as s:
        assert s.launches_per_step() == 3  # stress, velocity, record
        s.run(nt)
        tr, vz = s.seismograms(), s.field(F.F_VZ)
    assert np.abs(tr).max() > 0
    np.testing.assert_array_equal(tr[:, -1].reshape(2, n - 1, n - 1), np.stack([vz[1, 1:n, 1:n], vz[nz - 1, 1:n, 1:n]]))


@pytest.mark.parametrize("spacing", [(40.0, 10.0, 3.0), (9.1, 1.1, 10.3)])  # one and two correction steps
def test_fp64_division(cuda_device, spacing):
    m = I.random_small(F.MODEL_ORTHO, 33, 21, 17, nt=24, seed=8, damping=F.DAMP_SEPARABLE)
    m.dx, m.dy, m.dz = spacing
    m.dt = m.dt * min(spacing) / 12.0
    _check(m, 24, precision=F.PREC_F64)


@pytest.mark.parametrize("splits", [(7, 1, 8, 9, 25), (64 + 8 + 3, 16, 9), (1, 8, 64 + 16)])  # odd and even starts, graphs of 64 and of 8
@pytest.mark.parametrize("precision", [F.PREC_F32, F.PREC_F64])
def test_runs_in_graphs_and_single_steps(cuda_device, splits, precision):
    m = I.random_small(F.MODEL_ORTHO, 26, 19, 12, nt=sum(splits), seed=9, damping=F.DAMP_SEPARABLE)
    ref = O.run(m, m.nt, precision=precision)
    with Solver.from_model(m, precision=precision) as s:
        for n in splits:
            s.run(n)
        np.testing.assert_array_equal(s.seismograms(), ref.traces)
        for q in F.STATE:
            np.testing.assert_array_equal(s.field(q, ref.f[q].dtype), ref.f[q], err_msg=F.STATE_NAMES[q])
