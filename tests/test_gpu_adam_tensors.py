"""ewf_mlp_adam_all on tensors that its vector form does not take, among others that it does: the bits of ewf_mlp_adam."""
import ctypes as C

import pytest

from elanfmt_gb300.solver import load_library

pytestmark = pytest.mark.gpu
F = [C.c_float(v) for v in (1e-2, 0.9, 0.999, 1e-8)]


def _arrays(ts, wb):
    arr = lambda k: (C.c_void_p * len(ts))(*[t[k].data_ptr() for t in ts])  # noqa: E731
    return [arr(k) for k in range(4)] + [(C.c_void_p * len(ts))(*[x.data_ptr() if x is not None else None for x in wb])]


def test_views_into_one_buffer(cuda_device):
    import torch

    lib = load_library()
    g = torch.Generator(device="cuda").manual_seed(3)
    ns = [5, 128, 1027, 0, 4096, 3, 64, 1, 999] * 4
    flat = [torch.randn(sum(ns) + 1, generator=g, device="cuda") for _ in range(4)]
    flat[2].abs_()
    half = torch.zeros(sum(ns) + 1, dtype=torch.bfloat16, device="cuda")

    def views():
        ts, wb, at = [], [], 1
        for q, n in enumerate(ns):
            # every other one in memory of its own, aligned
            t = [x[at:at + n] if q % 2 else x[at:at + n].clone() for x in flat]
            wb.append(half[at:at + n] if q % 3 == 0 else None)
            ts.append(t)
            at += n
        return ts, wb

    keep = [x.clone() for x in flat]
    ts, wb = views()
    ref = [[x.clone() for x in t] for t in ts]
    refb = [None if x is None else torch.empty_like(x) for x in wb]
    for t, x in zip(ref, refb):
        if t[0].numel():
            assert lib.ewf_mlp_adam(*[C.c_void_p(y.data_ptr()) for y in t], C.c_void_p(x.data_ptr()) if x is not None else None, t[0].numel(),
                                    *F, 4, C.c_float(0.02), None) == 0
    a = _arrays(ts, wb)
    for k in range(4):  # an empty view has no address
        for q, n in enumerate(ns):
            if n == 0:
                a[k][q] = flat[k].data_ptr()
    assert lib.ewf_mlp_adam_all(len(ns), *a, (C.c_size_t * len(ns))(*ns), (C.c_float * len(ns))(*[0.02] * len(ns)), *F, 4, None) == 0
    torch.cuda.synchronize()
    for t, r, x, y in zip(ts, ref, wb, refb):
        assert all(torch.equal(p, q) for p, q in zip(t, r)) and (x is None or torch.equal(x, y))
    assert torch.equal(flat[3], keep[3]) and flat[0][0] == keep[0][0]


def test_parameters_that_are_views(cuda_device):
    """Weights as views into one buffer, as optimisers with flat parameters keep them."""
    import torch

    from elanfmt_gb300.surrogate import MLP

    a, b = MLP([128, 256, 128], seed=1), MLP([128, 256, 128], seed=1)
    flat = torch.zeros(sum(w.numel() for w in b.W) + 1, device="cuda")
    at = 1
    for l, w in enumerate(b.W):
        v = flat[at:at + w.numel()].view_as(w)
        v.copy_(w)
        b.W[l] = v
        at += w.numel()
    X, T = torch.randn(128, 128, device="cuda").to(torch.bfloat16), torch.randn(128, 128, device="cuda")
    for net in (a, b):
        net.forward(X)
        net.loss_grad(T)
        net.backward(128)
        net.adam(128, 1e-3)
    assert all(torch.equal(x, y) for x, y in zip(a.W + a.Wb + a.b, b.W + b.Wb + b.b))


def test_more_than_two_to_the_31_elements(cuda_device):
    import torch

    lib = load_library()
    n, edge = (1 << 31) + 3, 5000
    small = [torch.rand(edge, device="cuda") for _ in range(4)]
    big = [torch.zeros(n, device="cuda") for _ in range(4)]
    for s, x in zip(small, big):
        x[-edge:] = s
    ts = [small, big]
    sizes = (C.c_size_t * 2)(edge, n)
    assert lib.ewf_mlp_adam_all(2, *_arrays(ts, [None, None]), sizes, (C.c_float * 2)(0.0, 0.0), *F, 2, None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(s, x[-edge:]) for s, x in zip(small, big))
    assert not big[0][:edge].any()
