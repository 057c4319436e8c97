"""The two-kernel step from 0.4 M cells on, where FP32 runs two cells per thread (and from 1 to 6 M with streaming hints):
every scheme and option against the oracle, bit for bit, from a state that is random in every cell -- values of all
magnitudes down to the subnormals, zeros of both signs -- on odd and even extents."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(80, 70, 73), (79, 71, 75)]
STREAMED = (103, 99, 101)
NT = 7


def _state(m, seed, inf=False):
    rng = np.random.default_rng(seed)
    s = O.State(m, np.float32)
    for q in F.STATE:
        a = s.f[q]
        v = rng.normal(size=a.shape) * (1e-3 if q <= F.F_VZ else 1e4)
        kind = rng.random(a.shape)
        v = np.where(kind < 0.1, v * 10.0 ** rng.uniform(-40, 0, a.shape), v)  # small ones, subnormal results among them
        v = np.where(kind > 0.95, 0.0 * v, v)                                  # zeros of both signs
        v[v.shape[0] // 2:, :9] *= 1e-36                                       # a slab of quotients below 2^-90
        a[...] = v.astype(np.float32)
    if inf:
        s.f[F.F_VY][5, 6, 7] = np.inf
        s.f[F.F_SXX][9, 8, 30] = -np.inf
    return s


def _copy(s, m):
    c = O.State(m, np.float32)
    for q in F.STATE:
        c.f[q][...] = s.f[q]
    return c


def _check(m, precision=F.PREC_F32, seed=1, inf=False, settings=((0, 0, 0),)):
    assert m.nx * m.ny * m.nz >= 4e5
    init = _state(m, seed, inf)
    ref = _copy(init, m)
    if precision == F.PREC_F32_KAHAN:
        ref.comp = [np.zeros(F.shape(q, m.nx, m.ny, m.nz), np.float32) for q in (F.F_VX, F.F_VY, F.F_VZ)]
    with np.errstate(all="ignore"):
        O.run(m, NT, precision, ref)
    for kchunk, tile, prefetch in settings:
        with Solver.from_model(m, precision=precision, kchunk=kchunk, check_finite=False) as s:
            if tile:
                s.set_tile(tile)
                s.set_l2_prefetch(prefetch)
            for q in F.STATE:
                s.set_field(q, init.f[q])
            s.run(3)
            s.run(NT - 3)
            for q in F.STATE:
                got, want = s.field(q), ref.f[q]
                np.testing.assert_array_equal(got, want, err_msg=f"{F.STATE_NAMES[q]} {kchunk} {tile} {prefetch}")
                zero = want == 0
                np.testing.assert_array_equal(np.signbit(got[zero]), np.signbit(want[zero]), err_msg=f"zeros of {F.STATE_NAMES[q]}")
            np.testing.assert_array_equal(s.seismograms(), ref.traces, err_msg=f"{kchunk} {tile} {prefetch}")


def _model(model, shape, seed, nsrc=7, planes=(0, 1, 2, 3), **kw):
    m = I.random_small(model, *shape, nt=NT, seed=seed, **kw)
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    ent = [(c, i, j, k) for k in planes for c in (F.F_SXX, F.F_SZZ, F.F_SXY, F.F_SXZ, F.F_SYZ) for i, j in ((0, 5), (9, 0), (nx - 1, 7), (30, 31), (31, 31))]
    ent = [ent[q] for q in rng.permutation(len(ent))[:nsrc]]
    m.sources, m.source_coef = np.array(ent, np.int32), rng.normal(size=nsrc)
    m.receivers = np.array([(i, j, k, c) for i, j in ((1, 1), (2, 1), (3, 1), (32, 9), (33, 9), (nx - 2, 4), (nx - 1, ny - 1))
                            for k in (1, 2, 3, nz - 1) for c in range(3)], np.int32)
    return m


SCHEMES = [("iso", F.MODEL_ISO, {}), ("ortho-sep", F.MODEL_ORTHO, {"damping": F.DAMP_SEPARABLE}), ("ortho-w3d", F.MODEL_ORTHO, {"damping": F.DAMP_W3D}),
           ("isohet-sep", F.MODEL_ISO_HET, {"damping": F.DAMP_SEPARABLE}), ("isohet-w3d", F.MODEL_ISO_HET, {"damping": F.DAMP_W3D}),
           ("percomp", F.MODEL_ISO, {"damping": F.DAMP_PERCOMP})]  # (one cell per thread)
EACH = pytest.mark.parametrize("name,model,kw", SCHEMES, ids=[s[0] for s in SCHEMES])


@EACH
@pytest.mark.parametrize("precision", [F.PREC_F32, F.PREC_F32_KAHAN], ids=["f32", "kahan"])
@pytest.mark.parametrize("shape", SHAPES + [STREAMED], ids=lambda s: "x".join(map(str, s)))
def test_schemes(cuda_device, name, model, kw, precision, shape):
    _check(_model(model, shape, 11, **kw), precision)


@EACH
@pytest.mark.parametrize("order", [F.SRC_BEFORE_BC1, F.SRC_AFTER_BC1], ids=["before", "after"])
@pytest.mark.parametrize("nsrc,planes", [(30, (0, 1, 2, 3)), (7, (0, 2, 3)), (1, (1,))])  # in device memory, in the parameters, plane 1 alone
def test_sources(cuda_device, name, model, kw, order, nsrc, planes):
    if name == "percomp" and order == F.SRC_BEFORE_BC1:
        pytest.skip("that scheme injects after the boundary condition")
    _check(_model(model, SHAPES[1], 12, nsrc, planes, src_order=order, **kw))


@EACH
def test_launch_shapes(cuda_device, name, model, kw):
    """Tile heights, chunks and the velocity kernel's prefetch."""
    _check(_model(model, SHAPES[1], 13, **kw), settings=((4, 1, 1), (5, 2, 0), (7, 8, 2), (16, 16, 5), (64, 4, 3)))


@EACH
@pytest.mark.parametrize("precision", [F.PREC_F32, F.PREC_F32_KAHAN], ids=["f32", "kahan"])
@pytest.mark.parametrize("shape", [SHAPES[0], STREAMED], ids=lambda s: "x".join(map(str, s)))
def test_no_surface_condition(cuda_device, name, model, kw, precision, shape):
    m = _model(model, shape, 14, **kw)
    m.free_surface = F.FS_NONE
    if name == "iso":
        m.surface_mu = 1e-5
    _check(m, precision)


@pytest.mark.parametrize("precision", [F.PREC_F32, F.PREC_F32_KAHAN], ids=["f32", "kahan"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_surface_modulus(cuda_device, precision, shape):
    m = _model(F.MODEL_ISO, shape, 15)
    m.surface_mu = 2e3
    _check(m, precision)


@pytest.mark.parametrize("name,model,kw", SCHEMES[1:5], ids=[s[0] for s in SCHEMES[1:5]])
@pytest.mark.parametrize("shape", [SHAPES[1], STREAMED], ids=lambda s: "x".join(map(str, s)))
def test_velocity_damping(cuda_device, name, model, kw, shape):
    m = _model(model, shape, 16, **kw)
    m.vdamp = F.VDAMP_16KM
    _check(m)


@pytest.mark.parametrize("name,model,kw", SCHEMES[:5], ids=[s[0] for s in SCHEMES[:5]])
def test_infinities(cuda_device, name, model, kw):
    _check(_model(model, SHAPES[1], 17, **kw), inf=True)
