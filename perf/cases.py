"""Timed cases of the framework: what its users run, at sizes from a smoke test to the full grids.

Five kinds of work, each through the entry points a program calls:

* ``fdtd``     one solver handle: reset, run the time loop, read the seismograms and a snapshot
               component (`Solver`), over the models, precisions and damping forms;
* ``batch``    several right-hand sides and models advanced together (`Batch`): the elementary
               moment tensors of an inversion on one model, plus independent isotropic models;
* ``predict``  the learned Green's functions: network inference and the azimuthal mixing;
* ``train``    one training step of that network: forward, loss gradient, backward, Adam;
* ``filter``   the band-pass of device-resident seismograms (`sosfilt_device`).

`exact` restates each of them in plain 64-bit torch or numpy.
"""
import ctypes
import math

import numpy as np
import torch

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300 import postproc as P
from elanfmt_gb300 import surrogate as S
from elanfmt_gb300.solver import Batch, Solver, load_library

MODELS = {"iso": F.MODEL_ISO, "ortho": F.MODEL_ORTHO, "isohet": F.MODEL_ISO_HET}
PRECISIONS = {"f32": F.PREC_F32, "kahan": F.PREC_F32_KAHAN, "f64": F.PREC_F64}


def listed():
    return [
        # a first look at a new model: a small grid for a few steps, where launches and latency count
        dict(name="fdtd_ortho_40", kind="fdtd", model="ortho", nx=40, ny=40, nz=32, steps=60, precision="f32", damping="separable", tune=False),
        # the plain isotropic workload at its usual size (the fields almost fit the L2)
        dict(name="fdtd_iso_128", kind="fdtd", model="iso", nx=128, ny=128, nz=128, steps=1000, precision="f32", damping="pml", tune=False),
        # a station model with edge moduli and a 3-D sponge, odd extents, launch settings left alone
        dict(name="fdtd_isohet_ragged", kind="fdtd", model="isohet", nx=203, ny=151, nz=97, steps=400, precision="f32", damping="w3d", tune=False),
        # the full orthorhombic grid of the benchmark, launch settings autotuned once as it does
        dict(name="fdtd_ortho_320", kind="fdtd", model="ortho", nx=320, ny=320, nz=256, steps=400, precision="f32", damping="separable", tune=True),
        # the precision study's forms: compensated velocities, and the FP64 run both are measured against
        dict(name="fdtd_kahan_192", kind="fdtd", model="ortho", nx=192, ny=192, nz=192, steps=200, precision="kahan", damping="separable", tune=False),
        dict(name="fdtd_f64_128", kind="fdtd", model="ortho", nx=128, ny=128, nz=128, steps=100, precision="f64", damping="separable", tune=False),
        # a moment-tensor inversion's six elementary runs beside independent isotropic models
        dict(name="batch_6mt_6iso", kind="batch", n_ortho=128, rhs=6, n_iso=6, iso_lo=96, iso_hi=160, steps=100),
        # a few Green's-function queries (the batch is padded to a GEMM tile)
        dict(name="predict_100", kind="predict", queries=100, samples=1280, hidden=512, layers=4),
        # a catalogue of queries, in the study's batches
        dict(name="predict_8192", kind="predict", queries=8192, samples=1024, hidden=512, layers=4),
        # a training step of the structured network at the study's minibatch, and of the 18-trace form at a larger one
        dict(name="train_256", kind="train", batch=256, traces=10, samples=1024, hidden=512, layers=4),
        dict(name="train_1024_full", kind="train", batch=1024, traces=18, samples=1024, hidden=512, layers=4),
        # the driver's band-pass over a run's receivers
        dict(name="filter_192", kind="filter", traces=192, samples=4000, sections=4),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fdtd", "fdtd", "fdtd", "fdtd", "batch", "predict", "train", "filter"])
    if kind == "fdtd":
        model = rng.choice(["iso", "ortho", "isohet"])
        precision = rng.choice(["f32", "f32", "f32", "kahan", "f64"])
        top = 256 if precision != "f64" else 128
        return dict(kind="fdtd", model=model, nx=_log(rng, 36, top), ny=_log(rng, 36, top), nz=_log(rng, 32, top),
                    steps=_log(rng, 60, 400 if precision != "f64" else 100), precision=precision,
                    damping="pml" if model == "iso" else rng.choice(["separable", "w3d"]), tune=rng.random() < 0.25)
    if kind == "batch":
        lo = _log(rng, 48, 96)
        return dict(kind="batch", n_ortho=_log(rng, 48, 144), rhs=rng.choice([1, 3, 6, 6]), n_iso=rng.randint(1, 6),
                    iso_lo=lo, iso_hi=lo + rng.randint(8, 56), steps=_log(rng, 40, 100))
    if kind == "predict":
        return dict(kind="predict", queries=_log(rng, 1, 8192), samples=128 * rng.randint(2, 10), hidden=512, layers=4)
    if kind == "train":
        return dict(kind="train", batch=128 * _log(rng, 1, 8), traces=rng.choice([10, 18]), samples=128 * rng.randint(2, 8),
                    hidden=rng.choice([256, 512]), layers=rng.randint(3, 4))
    return dict(kind="filter", traces=_log(rng, 3, 3000), samples=_log(rng, 500, 6000), sections=rng.choice([2, 4, 4, 6]))


# ---------------------------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------------------------

def _layered(c, seed):
    """A horizontally layered model of the case's scheme: layers, source mechanism and wavelet from
    the seed; the edge moduli and buoyancies are those means of equal neighbours inside a layer."""
    nx, ny, nz, steps = c["nx"], c["ny"], c["nz"], c["steps"]
    rng = np.random.default_rng(seed)
    layers = I.layered_ortho_layers(8, int(rng.integers(1 << 30)))
    li = I.layer_index(nz, 8)
    prof = {k: np.array([layers[q][k] for q in li]) for k in layers[0]}
    if c["model"] != "ortho":  # isotropic: vp and vs of the layer's C33 and C55
        for k in ("C11", "C22"):
            prof[k] = prof["C33"]
        prof["C44"] = prof["C66"] = prof["C55"]
        prof["C12"] = prof["C33"] - 2 * prof["C55"]
    vmax = math.sqrt(float(np.max(np.maximum(np.maximum(prof["C11"], prof["C22"]), prof["C33"]) / prof["rho"])))
    vmin = math.sqrt(float(np.min(prof["C55"] / prof["rho"])))
    dx = 40.0
    m = I.Model(nx=nx, ny=ny, nz=nz, nt=steps, dx=dx, dy=dx, dz=dx, dt=float(np.float32(0.5 * dx / (vmax * math.sqrt(3.0)))),
                model=MODELS[c["model"]], damping=F.DAMP_PML1D)

    def cells(v):
        return np.ascontiguousarray(np.broadcast_to(v.astype(np.float32)[:, None, None], (nz, ny, nx)))

    def edges(v, plane):
        out = np.zeros(F.shape({"xy": F.M_C66XY, "xz": F.M_C55XZ, "yz": F.M_C44YZ}[plane], nx, ny, nz), np.float32)
        if plane == "xy":
            out[:, 1:-1, 1:-1] = v[:, None, None]
        else:
            out[1:-1] = (2.0 / (1.0 / v[:-1] + 1.0 / v[1:]))[:, None, None]
            if plane == "xz":
                out[:, :, 0] = out[:, :, -1] = 0
            else:
                out[:, 0] = out[:, -1] = 0
        return out

    def faces(b, axis):
        out = np.zeros(F.shape({"x": F.M_BX, "y": F.M_BY, "z": F.M_BZ}[axis], nx, ny, nz), np.float32)
        if axis == "x":
            out[:, :, 1:-1] = b[:, None, None]
        elif axis == "y":
            out[:, 1:-1, :] = b[:, None, None]
        else:
            out[1:-1] = (0.5 * (b[:-1] + b[1:]))[:, None, None]
        return out

    b = 1.0 / prof["rho"]
    lpml = max(4, min(15, min(nx, ny, nz) // 6))
    if c["model"] == "iso":
        # cell fields c11, c12 with a few per cent of scatter; mu and 1/rho are scalars of this scheme
        scatter = rng.uniform(0.97, 1.0, size=(nz, ny, nx)).astype(np.float32)
        m.materials[F.M_C11] = cells(prof["C11"]) * scatter
        m.materials[F.M_C12] = cells(prof["C12"]) * scatter
        m.c66 = float(np.float32(np.min(prof["C55"])))
        m.bx = m.by = m.bz = float(np.float32(np.min(b)))
        m.src_order = F.SRC_BEFORE_BC1
        for fid, n in ((F.D_WX, nx), (F.D_WY, ny), (F.D_WZ, nz)):
            m.damping_arrays[fid] = I.pml_weights(n, lpml, m.dt)
    else:
        m.src_order = F.SRC_AFTER_BC1
        ids = {"C11": F.M_C11, "C12": F.M_C12}
        if c["model"] == "ortho":
            ids.update({"C22": F.M_C22, "C33": F.M_C33, "C13": F.M_C13, "C23": F.M_C23})
        for k, fid in ids.items():
            m.materials[fid] = cells(prof[k])
        m.materials[F.M_C66XY] = edges(prof["C66"], "xy")
        m.materials[F.M_C55XZ] = edges(prof["C55"], "xz")
        m.materials[F.M_C44YZ] = edges(prof["C44"], "yz")
        m.materials[F.M_BX], m.materials[F.M_BY], m.materials[F.M_BZ] = faces(b, "x"), faces(b, "y"), faces(b, "z")
        w = [I.pml_factors(n, lpml, m.dt, sides=s) for n, s in ((nx, "both"), (ny, "both"), (nz, "high"))]
        if c["damping"] == "w3d":
            m.damping = F.DAMP_W3D
            m.damping_arrays[F.D_W3D] = I.separable_weights(*w)
        else:
            m.damping = F.DAMP_SEPARABLE
            for fid, a in zip((F.D_WX, F.D_WY, F.D_WZ), w):
                m.damping_arrays[fid] = a
    mt, _ = I.lune_moment_tensor(int(rng.integers(1 << 30)))
    zs = max(6, nz // 4)
    m.set_moment_tensor(mt, nx // 2 - 1, ny // 2 - 1, zs - 1, stencil=0 if c["model"] == "iso" else 1)
    f0 = vmin / (float(rng.uniform(9, 11)) * dx)
    m.stf = I.ricker_stf(steps, m.dt, f0, scale=1e15 / dx ** 3)
    # an 8 x 8 surface spread and a string down through the source's depth, three components each
    at = lambda n: [int(round(v)) for v in np.linspace(0.15 * n, 0.85 * n, 8)]  # noqa: E731
    rec = [(i, j, 1, q) for j in at(ny) for i in at(nx) for q in range(3)]
    rec += [(nx // 2 + 3, ny // 2 - 2, k, q) for k in range(2, nz - 2, max(1, nz // 8)) for q in range(3)]
    m.receivers = np.array(rec, np.int32)
    return m


def _batch_problems(c, seed):
    """(model, [(sources, coefficients) per right-hand side]) of each problem."""
    n = c["n_ortho"]
    m = _layered(dict(model="ortho", damping="separable", nx=n, ny=n, nz=n, steps=c["steps"]), seed)
    xs, ys, zs = (int(v) - 1 for v in m.sources[0, 1:4])
    problems = [(m, [F.mt_entries(np.eye(6)[q], xs, ys, zs, 1) for q in range(c["rhs"])])]
    rng = np.random.default_rng([seed, 1])
    sizes = np.random.default_rng(c["n_ortho"] * 1000 + c["iso_lo"]).integers(c["iso_lo"], c["iso_hi"] + 1, size=c["n_iso"])
    for s in sizes:
        s = int(s)
        mi = _layered(dict(model="iso", damping="pml", nx=s, ny=s, nz=s, steps=c["steps"]), int(rng.integers(1 << 30)))
        problems.append((mi, [(mi.sources, mi.source_coef)]))
    return problems


# ---------------------------------------------------------------------------------------------
# network inputs
# ---------------------------------------------------------------------------------------------

def _net(c, seed):
    nout = c["samples"] * (S.NFUND if c["kind"] == "predict" else c["traces"])
    nin = 2 if c["kind"] == "predict" or c["traces"] == S.NFUND else 8
    net = S.MLP([S.IN_PAD] + [c["hidden"]] * c["layers"] + [nout], seed=seed, fan_in0=nin)
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows = c["queries"] if c["kind"] == "predict" else c["batch"]
    X = torch.zeros(rows, S.IN_PAD, device="cuda")
    X[:, :nin] = torch.randn(rows, nin, generator=g, device="cuda")
    return net, X.to(torch.bfloat16), g


def _train_state(c, seed):
    """A network in mid-training: Adam's moments have history."""
    net, X, g = _net(c, seed)
    T = torch.randn(c["batch"], net.sizes[-1], generator=g, device="cuda")
    net.step_count = 500
    for w, m, v in list(zip(net.W, net.mW, net.vW)) + list(zip(net.b, net.mb, net.vb)):
        m.copy_(1e-5 * torch.randn(w.shape, generator=g, device="cuda"))
        v.copy_(1e-9 * (0.5 + torch.rand(w.shape, generator=g, device="cuda")))
    return net, X, T


LR = 5e-4


def _filter_inputs(c, seed):
    sos = P.butter_bandpass(c["sections"], 1 / 2.5, 1 / 0.5, 1 / 2.4056e-3)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(c["traces"], c["samples"], generator=g, device="cuda", dtype=torch.float64).cumsum(1)
    return sos, x


def _queries_mixing(c, seed):
    return torch.from_numpy(S.mixing_matrices(np.random.default_rng(seed).uniform(-math.pi, math.pi, c["queries"]))).cuda()


# ---------------------------------------------------------------------------------------------
# the contract: prepare, run, work, exact
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    if k == "fdtd":
        s = Solver.from_model(_layered(case, seed), precision=PRECISIONS[case["precision"]])
        if case["tune"]:
            s.autotune(min(10, case["steps"] - 1))
        return dict(kind=k, solver=s, steps=case["steps"], dtype=np.float64 if case["precision"] == "f64" else np.float32)
    if k == "batch":
        return dict(kind=k, batch=Batch(_batch_problems(case, seed)), steps=case["steps"])
    if k == "predict":
        net, X, _ = _net(case, seed)
        return dict(kind=k, net=net, X=X, R=_queries_mixing(case, seed), samples=case["samples"], lib=load_library())
    if k == "train":
        net, X, T = _train_state(case, seed)
        return dict(kind=k, net=net, X=X, T=T)
    sos, x = _filter_inputs(case, seed)
    return dict(kind=k, sos=sos, x=x)


def run(state):
    k = state["kind"]
    if k == "fdtd":
        s = state["solver"]
        s.reset()
        s.run(state["steps"])
        return {"traces": s.seismograms(), "vz": s.field(F.F_VZ, dtype=state["dtype"])}
    if k == "batch":
        b = state["batch"]
        b.reset()
        b.run(state["steps"])
        return {f"{p}.{r}": b.seismograms(p, r) for p in range(len(b.models)) for r in range(b.nrhs[p])}
    if k == "predict":
        y = state["net"].predict(state["X"])
        n, t = len(y), state["samples"]
        out = torch.empty(n, S.NCOMP * t, device="cuda")
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
        if state["lib"].ewf_mlp_combine(p(state["R"]), p(y), p(out), n, S.NCOMP, S.NFUND, t, stream):
            raise RuntimeError("ewf_mlp_combine")
        return {"fundamentals": y, "traces": out}
    if k == "train":
        net, X, T = state["net"], state["X"], state["T"]
        net.forward(X)
        loss = net.loss_grad(T)
        net.backward(len(X))
        net.adam(len(X), LR)
        return {"loss": loss, "W": net.W, "b": net.b, "mW": net.mW, "vW": net.vW, "mb": net.mb, "vb": net.vb}
    t = state["x"].clone()
    P.sosfilt_device(state["sos"], t)
    return t


def _fdtd_work(model, precision, cells, steps, damping):
    # compulsory bytes of a step: nine state fields read and written, the material fields read (iso 2,
    # isohet 8, ortho 12) and a 3-D damping field where there is one; FP64 doubles all of them
    b = 72 + 4 * {"iso": 2, "isohet": 8, "ortho": 12}[model] + (4 if damping == "w3d" else 0)
    b = {"f32": b, "kahan": b + 24, "f64": 2 * b}[precision]
    return cells * steps * b, cells * steps * {"iso": 82, "isohet": 92, "ortho": 98}[model]


def work(case):
    k = case["kind"]
    if k == "fdtd":
        byts, flops = _fdtd_work(case["model"], case["precision"], case["nx"] * case["ny"] * case["nz"], case["steps"], case["damping"])
        return {"bytes": byts, "flops": flops}
    if k == "batch":
        n = case["n_ortho"] ** 3
        # the right-hand sides share the model: its 12 fields are read once a step
        byts = case["steps"] * n * (48 + 72 * case["rhs"])
        flops = case["steps"] * n * 98 * case["rhs"]
        sizes = np.random.default_rng(case["n_ortho"] * 1000 + case["iso_lo"]).integers(case["iso_lo"], case["iso_hi"] + 1, size=case["n_iso"])
        for s in sizes:
            b, f = _fdtd_work("iso", "f32", int(s) ** 3, case["steps"], "pml")
            byts, flops = byts + b, flops + f
        return {"bytes": byts, "flops": flops}
    if k in ("predict", "train"):
        nout = case["samples"] * (S.NFUND if k == "predict" else case["traces"])
        rows = case["queries"] if k == "predict" else case["batch"]
        sizes = [S.IN_PAD] + [case["hidden"]] * case["layers"] + [nout]
        weights = sum(a * b for a, b in zip(sizes, sizes[1:]))
        if k == "predict":  # bf16 weights and inputs, the fundamental traces written, the mixed traces written
            mix = rows * S.NCOMP * S.NFUND
            return {"bytes": 2 * weights + 2 * rows * S.IN_PAD + 4 * rows * nout + 4 * mix + 4 * rows * S.NCOMP * case["samples"],
                    "flops": 2 * rows * weights + 2 * mix * case["samples"]}
        # fp32 weight and two moments read and written, bf16 weights read and written, the targets read
        return {"bytes": 28 * weights + 4 * rows * nout + 2 * rows * S.IN_PAD, "flops": 6 * rows * weights}
    n = case["traces"] * case["samples"]
    return {"bytes": 16 * n, "flops": 9 * case["sections"] * n}


def _fdtd_exact(m, sources, coef):
    """The scheme in FP64 torch: every field with a zero margin, cell (i, j, k) at [k+1, j+1, i+1]."""
    nx, ny, nz = m.nx, m.ny, m.nz
    f = [torch.zeros(nz + 3, ny + 3, nx + 3, dtype=torch.float64, device="cuda") for _ in range(9)]
    vx, vy, vz, sxx, syy, szz, sxy, sxz, syz = f
    mat = {q: torch.from_numpy(a).cuda()[:nz, :ny, :nx].double() for q, a in m.materials.items()}
    d = {q: torch.from_numpy(a).cuda().double() for q, a in m.damping_arrays.items()}
    dt, dx, dy, dz = m.dt, m.dx, m.dy, m.dz

    def at(a, k0, j0, i0, k1=nz, j1=ny, i1=nx, dk=0, dj=0, di=0):
        return a[k0 + 1 + dk:k1 + 1 + dk, j0 + 1 + dj:j1 + 1 + dj, i0 + 1 + di:i1 + 1 + di]

    iso = m.model == F.MODEL_ISO
    ax = lambda v, n: v.view([-1 if q == n else 1 for q in range(3)])  # noqa: E731
    if iso:
        wx, wy, wz = ax(d[F.D_WX], 2), ax(d[F.D_WY], 1), ax(d[F.D_WZ], 0)
        hx, hy, hz = 0.5 * (wx[..., 1:] + wx[..., :-1]), 0.5 * (wy[:, 1:] + wy[:, :-1]), 0.5 * (wz[1:] + wz[:-1])
        wxi, wyj, wzk = wx[..., :nx], wy[:, :ny], wz[:nz]
        wsh = wxi * wyj * wzk
        c11 = c22 = c33 = mat[F.M_C11]
        c12 = c13 = c23 = mat[F.M_C12]
        g66 = g55 = g44 = m.c66
    else:
        if m.damping == F.DAMP_W3D:
            W = d[F.D_W3D]
        else:
            W = (ax(d[F.D_WX], 2) * ax(d[F.D_WY], 1)) * ax(d[F.D_WZ], 0)
        c11, c12 = mat[F.M_C11], mat[F.M_C12]
        if m.model == F.MODEL_ORTHO:
            c22, c33, c13, c23 = mat[F.M_C22], mat[F.M_C33], mat[F.M_C13], mat[F.M_C23]
        else:
            c22 = c33 = c11
            c13 = c23 = c12
        g66, g55, g44 = mat[F.M_C66XY], mat[F.M_C55XZ], mat[F.M_C44YZ]
    rows = min(nx, ny)
    rec = torch.from_numpy(np.asarray(m.receivers, np.int64)).cuda()
    tr = torch.zeros(len(rec), m.nt, dtype=torch.float64, device="cuda")
    by_comp = [(torch.nonzero(rec[:, 3] == q)[:, 0], rec[rec[:, 3] == q]) for q in range(3)]
    for it in range(m.nt):
        c = lambda a, **o: at(a, 0, 0, 0, **o)  # noqa: E731
        exx = (c(vx, di=1) - c(vx)) / dx
        eyy = (c(vy, dj=1) - c(vy)) / dy
        ezz = (c(vz, dk=1) - c(vz)) / dz
        exy = (c(vy) - c(vy, di=-1)) / dx + (c(vx) - c(vx, dj=-1)) / dy
        exz = (c(vz) - c(vz, di=-1)) / dx + (c(vx) - c(vx, dk=-1)) / dz
        eyz = (c(vy) - c(vy, dk=-1)) / dz + (c(vz) - c(vz, dj=-1)) / dy
        nxx, nyy, nzz = c11 * exx + c12 * eyy + c13 * ezz, c12 * exx + c22 * eyy + c23 * ezz, c13 * exx + c23 * eyy + c33 * ezz
        if iso:
            c(sxx).add_(nxx, alpha=dt).mul_(hx)
            c(syy).add_(nyy, alpha=dt).mul_(hy)
            c(szz).add_(nzz, alpha=dt).mul_(hz)
            for s, e in ((sxy, exy), (sxz, exz), (syz, eyz)):
                c(s).add_(e, alpha=dt * g66).mul_(wsh)
        else:
            for s, e in ((sxx, nxx), (syy, nyy), (szz, nzz)):
                c(s).mul_(W).add_(e, alpha=dt)
            W_, g = (W[:, 1:, 1:], W[1:, :, 1:], W[1:, 1:, :]), (g66[:, 1:, 1:], g55[1:, :, 1:], g44[1:, 1:, :])
            at(sxy, 0, 1, 1).mul_(W_[0]).add_(g[0] * exy[:, 1:, 1:], alpha=dt)
            at(sxz, 1, 0, 1).mul_(W_[1]).add_(g[1] * exz[1:, :, 1:], alpha=dt)
            at(syz, 1, 1, 0).mul_(W_[2]).add_(g[2] * eyz[1:, 1:, :], alpha=dt)
        # the sources lie below the planes of the free-surface rule, so their order does not matter here
        at(szz, 0, 0, 0, k1=1, j1=rows).zero_()
        at(sxz, 1, 0, 1, k1=2, j1=rows).copy_(at(sxz, 2, 0, 1, k1=3, j1=rows) / 3)
        at(syz, 1, 1, 0, k1=2).copy_(at(syz, 2, 1, 0, k1=3) / 3)
        for (q, i, j, k), a in zip(sources, coef):
            f[q][k + 1, j + 1, i + 1] += float(a) * float(m.stf[it])
        for v, (k1, j1, i1), w in ((vx, (nz - 1, ny - 1, nx), 0), (vy, (nz - 1, ny, nx - 1), 1), (vz, (nz, ny - 1, nx - 1), 2)):
            s = lambda a, **o: at(a, 1, 1, 1, k1, j1, i1, **o)  # noqa: E731
            if w == 0:
                div = (s(sxx) - s(sxx, di=-1)) / dx + (s(sxy, dj=1) - s(sxy)) / dy + (s(sxz, dk=1) - s(sxz)) / dz
            elif w == 1:
                div = (s(syy) - s(syy, dj=-1)) / dy + (s(sxy, di=1) - s(sxy)) / dx + (s(syz, dk=1) - s(syz)) / dz
            else:
                div = (s(szz) - s(szz, dk=-1)) / dz + (s(sxz, di=1) - s(sxz)) / dx + (s(syz, dj=1) - s(syz)) / dy
            if iso:
                damp = (wx[..., :i1 - 1], wy[:, :j1 - 1], wz[:k1 - 1])[w]
                s(v).add_(div, alpha=dt * (m.bx, m.by, m.bz)[w]).mul_(damp)
            else:
                b = (mat[F.M_BX], mat[F.M_BY], mat[F.M_BZ])[w][1:k1, 1:j1, 1:i1]
                s(v).mul_(W[1:k1, 1:j1, 1:i1]).add_(b * div, alpha=dt)
        for q, (at_q, r) in enumerate(by_comp):
            tr[at_q, it] = f[q][r[:, 2] + 1, r[:, 1] + 1, r[:, 0] + 1]
    return tr.cpu().numpy(), at(vz, 0, 0, 0, k1=nz + 1).cpu().numpy()


def _forward64(net, X):
    """Pre-activations and activations of the network in 64 bits, from its bf16 weights."""
    h, pre, act = X.double(), [], [X.double()]
    for q, (w, b) in enumerate(zip(net.Wb, net.b)):
        p = h @ w.double().T + b.double()
        h = torch.nn.functional.gelu(p) if q < len(net.Wb) - 1 else p
        pre.append(p)
        act.append(h)
    return pre, act


def exact(case, seed):
    k = case["kind"]
    if k == "fdtd":
        m = _layered(case, seed)
        tr, vz = _fdtd_exact(m, m.sources, m.source_coef)
        return {"traces": tr, "vz": vz}
    if k == "batch":
        return {f"{p}.{r}": _fdtd_exact(m, e, a)[0] for p, (m, rhs) in enumerate(_batch_problems(case, seed))
                for r, (e, a) in enumerate(rhs)}
    if k == "predict":
        net, X, _ = _net(case, seed)
        R, t = _queries_mixing(case, seed).double(), case["samples"]
        y = torch.cat([_forward64(net, x)[1][-1] for x in X.split(1024)])
        out = torch.cat([torch.bmm(r, g.view(-1, S.NFUND, t)).view(len(r), -1) for r, g in zip(R.split(1024), y.split(1024))])
        return {"fundamentals": y, "traces": out}
    if k == "train":
        net, X, T = _train_state(case, seed)
        pre, act = _forward64(net, X)
        d = (act[-1] - T.double()) * (2.0 / T.numel())
        out = {"loss": ((act[-1] - T.double()) ** 2).mean(), "W": [], "b": [], "mW": [], "vW": [], "mb": [], "vb": []}
        gW, gb = [], []
        for q in range(net.nlayers - 1, -1, -1):
            gW.insert(0, d.T @ act[q])
            gb.insert(0, d.sum(0))
            if q:
                p = pre[q - 1]
                grad = 0.5 * (1 + torch.erf(p / math.sqrt(2.0))) + p * torch.exp(-0.5 * p * p) / math.sqrt(2 * math.pi)
                d = (d @ net.Wb[q].double()) * grad
        b1, b2, eps, n = 0.9, 0.999, 1e-8, net.step_count + 1
        for key, ws, ms, vs, gs in (("W", net.W, net.mW, net.vW, gW), ("b", net.b, net.mb, net.vb, gb)):
            for w, m, v, g in zip(ws, ms, vs, gs):
                m, v = b1 * m.double() + (1 - b1) * g, b2 * v.double() + (1 - b2) * g * g
                out[key].append(w.double() - LR * (m / (1 - b1 ** n)) / ((v / (1 - b2 ** n)).sqrt() + eps))
                out["m" + key].append(m)
                out["v" + key].append(v)
        return out
    sos, x = _filter_inputs(case, seed)
    # the sections as one recursion over time, every trace at once
    x = x.T.cpu().numpy()
    s1, s2 = np.zeros((len(sos), x.shape[1])), np.zeros((len(sos), x.shape[1]))
    y = np.empty_like(x)
    for t in range(len(x)):
        v = x[t]
        for q, (b0, b1, b2, a0, a1, a2) in enumerate(sos):
            o = b0 / a0 * v + s1[q]
            s1[q] = b1 / a0 * v - a1 / a0 * o + s2[q]
            s2[q] = b2 / a0 * v - a2 / a0 * o
            v = o
        y[t] = v
    return np.ascontiguousarray(y.T)
