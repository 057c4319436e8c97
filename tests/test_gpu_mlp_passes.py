"""The network's one-call passes (ewf_mlp_forward, _backward, _mse_loss, _adam_all) against the same work
done kernel by kernel (ewf_mlp_gemm, _transpose, _gelu_grad, ...): equal bit for bit where the sums keep
their order, within fp32 rounding for the bias gradients and the loss."""
import ctypes as C

import pytest

from elanfmt_gb300.solver import EwfError, load_library

pytestmark = pytest.mark.gpu


def p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


NETS = [[128, 128], [128, 256, 128], [256, 128, 384, 640], [128, 512, 512, 512, 512, 2560], [128] * 11]


@pytest.mark.parametrize("sizes", NETS, ids=lambda s: "-".join(map(str, s)))
@pytest.mark.parametrize("M", [128, 384, 1024])
def test_backward_equals_its_kernels(cuda_device, sizes, M):
    import torch

    from elanfmt_gb300.surrogate import MLP

    lib = load_library()
    net = MLP(sizes, seed=len(sizes))
    g = torch.Generator(device="cuda").manual_seed(M)
    X = torch.randn(M, sizes[0], generator=g, device="cuda").to(torch.bfloat16)
    T = torch.randn(M, sizes[-1], generator=g, device="cuda")
    Y = net.forward(X)
    loss = net.loss_grad(T)
    net.backward(M)
    w = net._work(M)
    assert lib.ewf_mlp_status() == 0
    # the forward pass layer by layer
    H = [X]
    for l in range(net.nlayers):
        last = l == net.nlayers - 1
        out = torch.empty(M, sizes[l + 1], device="cuda", dtype=torch.float32 if last else torch.bfloat16)
        pre = None if last else torch.empty(M, sizes[l + 1], device="cuda")
        assert lib.ewf_mlp_gemm(p(H[l]), p(net.Wb[l]), p(net.b[l]), p(out) if last else None, None if last else p(out), p(pre), M,
                                sizes[l + 1], sizes[l], 0 if last else 1, None) == 0
        if not last:
            assert torch.equal(out, w["H"][l + 1]) and torch.equal(pre, w["P"][l])
        H.append(out)
    assert torch.equal(H[-1], Y)
    # the loss and its gradient
    dy, part = torch.empty(M, sizes[-1], dtype=torch.bfloat16, device="cuda"), torch.empty(1024, device="cuda")
    assert lib.ewf_mlp_mse_grad(p(Y), p(T), p(dy), Y.numel(), C.c_float(1.0 / Y.numel()), p(part), 1024, None) == 0
    assert torch.equal(dy, w["dY"][-1])
    exact = ((Y.double() - T.double()) ** 2).mean()
    assert abs(float(loss) - float(exact)) < 1e-6 * float(exact)  # fp32 sums of non-negative terms in a tree
    # the gradients layer by layer, from transposed copies
    for l in range(net.nlayers - 1, -1, -1):
        nout, nin = sizes[l + 1], sizes[l]
        dyt, ht, gw = (torch.empty(nout, M, dtype=torch.bfloat16, device="cuda"), torch.empty(nin, M, dtype=torch.bfloat16, device="cuda"),
                       torch.empty(nout, nin, device="cuda"))
        assert lib.ewf_mlp_transpose(p(dy), p(dyt), M, nout, None) == 0 and lib.ewf_mlp_transpose(p(H[l]), p(ht), M, nin, None) == 0
        assert lib.ewf_mlp_gemm(p(dyt), p(ht), None, p(gw), None, None, nout, nin, M, 0, None) == 0
        assert torch.equal(gw, w["gW"][l]), f"layer {l}"
        db = dy.double().sum(0)
        # M rounded additions at most, on sums of at most sum |dy|
        assert ((w["gb"][l].double() - db).abs() <= 1.2e-7 * (M / 32 + 32) * dy.double().abs().sum(0)).all()
        if l:
            wt, dh = torch.empty(nin, nout, dtype=torch.bfloat16, device="cuda"), torch.empty(M, nin, dtype=torch.bfloat16, device="cuda")
            assert lib.ewf_mlp_transpose(p(net.Wb[l]), p(wt), nout, nin, None) == 0
            assert lib.ewf_mlp_gemm(p(dy), p(wt), None, None, p(dh), None, M, nin, nout, 0, None) == 0
            dy = torch.empty_like(dh)
            assert lib.ewf_mlp_gelu_grad(p(dh), p(w["P"][l - 1]), p(dy), dh.numel(), None) == 0
            assert torch.equal(dy, w["dY"][l - 1]), f"layer {l}"


@pytest.mark.parametrize("n", [1, 31, 33, 100, 129, 513])
def test_predict_any_row_count(cuda_device, n):
    import torch

    from elanfmt_gb300.surrogate import MLP

    net = MLP([128, 256, 512, 384], seed=5)
    X = torch.randn(640, 128, device="cuda").to(torch.bfloat16)
    whole = net.forward(X).clone()
    assert torch.equal(net.predict(X[:n]), whole[:n])
    assert torch.equal(net.predict(X[:n], batch=100), whole[:n])
    assert torch.equal(net.predict(X[1:n + 1].float()), whole[1:n + 1])          # converted, as the copy did
    wide = torch.zeros(n, 256, dtype=torch.bfloat16, device="cuda")
    wide[:, 3:131] = X[:n]
    assert torch.equal(net.predict(wide[:, 3:131]), whole[:n])                   # neither contiguous nor aligned
    with pytest.raises(EwfError):
        net.forward(X[:n])


def test_adam_all_equals_adam(cuda_device):
    import torch

    lib = load_library()
    ns = [1, 3, 4, 1023, 1024, 1025, 70000, 5, 8, 128, 131, 64, 2, 7, 12, 100, 33, 6]  # two groups, tails
    g = torch.Generator(device="cuda").manual_seed(0)
    one, all_ = [], []
    for n in ns:
        t = [torch.randn(n, generator=g, device="cuda") for _ in range(4)]
        t[2].abs_()
        one.append([x.clone() for x in t] + [torch.empty(n, dtype=torch.bfloat16, device="cuda") if n % 2 else None])
        all_.append([x.clone() for x in t] + [torch.empty(n, dtype=torch.bfloat16, device="cuda") if n % 2 else None])
    wd = [0.0 if q % 3 else 0.01 for q in range(len(ns))]
    f = [C.c_float(v) for v in (1e-2, 0.9, 0.999, 1e-8)]
    for (w, m, v, gr, wb), d in zip(one, wd):
        assert lib.ewf_mlp_adam(p(w), p(m), p(v), p(gr), p(wb), w.numel(), *f, 7, C.c_float(d), None) == 0
    arr = lambda k: (C.c_void_p * len(ns))(*[t[k].data_ptr() if t[k] is not None else None for t in all_])  # noqa: E731
    assert lib.ewf_mlp_adam_all(len(ns), arr(0), arr(1), arr(2), arr(3), arr(4), (C.c_size_t * len(ns))(*ns), (C.c_float * len(ns))(*wd), *f,
                                7, None) == 0
    torch.cuda.synchronize()
    for a, b in zip(one, all_):
        for x, y in zip(a, b):
            assert x is None or torch.equal(x, y)
