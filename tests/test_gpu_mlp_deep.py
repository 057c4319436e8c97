"""A network of more layers than a launch's tables hold: its passes against the work layer by layer."""
import ctypes as C

import pytest

from elanfmt_gb300.solver import load_library

pytestmark = pytest.mark.gpu


def p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def test_seventy_layers(cuda_device):
    import torch

    from elanfmt_gb300.surrogate import MLP

    lib = load_library()
    M, L = 128, 70
    net = MLP([128] * (L + 1), seed=2)
    X = torch.randn(M, 128, device="cuda").to(torch.bfloat16)
    Y = net.forward(X).clone()
    H = X
    for l in range(L):
        last = l == L - 1
        out = torch.empty(M, 128, device="cuda", dtype=torch.float32 if last else torch.bfloat16)
        assert lib.ewf_mlp_gemm(p(H), p(net.Wb[l]), p(net.b[l]), p(out) if last else None, None if last else p(out), None, M, 128, 128,
                                0 if last else 1, None) == 0
        H = out
    assert torch.equal(H, Y) and torch.equal(net.predict(X[:77]), Y[:77])
    T = torch.randn(M, 128, device="cuda")
    net.loss_grad(T)
    net.backward(M)
    w = net._work(M)
    for l in range(L):  # fp32 sums of M products, however small the gradient has become on its way
        exact = w["dY"][l].double().T @ w["H"][l].double()
        bound = w["dY"][l].double().abs().T @ w["H"][l].double().abs()
        assert exact.abs().max() > 0 and ((w["gW"][l].double() - exact).abs() <= 1.2e-7 * M * bound + 1e-44).all(), l
        db = w["dY"][l].double()
        assert ((w["gb"][l].double() - db.sum(0)).abs() <= 1.2e-7 * M * db.abs().sum(0) + 1e-44).all(), l
    grads = [(g.clone(), gb.clone()) for g, gb in zip(w["gW"], w["gb"])]
    mine = [(net.W[l].clone(), net.b[l].clone()) for l in range(L)]
    net.adam(M, 1e-3)
    f = [C.c_float(v) for v in (1e-3, 0.9, 0.999, 1e-8)]
    for l in range(L):
        for k, (x, g) in enumerate(zip(mine[l], grads[l])):
            m, v = torch.zeros_like(x), torch.zeros_like(x)
            assert lib.ewf_mlp_adam(p(x), p(m), p(v), p(g), None, x.numel(), *f, 1, C.c_float(0.0), None) == 0
            assert torch.equal(x, (net.W, net.b)[k][l]), l
    net.check_status()
