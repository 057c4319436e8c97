"""Inference of different batch sizes by one network from two threads, each on a stream of its own."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_predictions_that_overlap(cuda_device):
    import torch

    from elanfmt_gb300.surrogate import MLP

    net = MLP([128, 512, 512, 512, 512, 1280], seed=4)
    sizes = (8192, 1024)
    X = [torch.randn(n, 128, device="cuda").to(torch.bfloat16) for n in sizes]
    want = [net.predict(x).clone() for x in X]
    torch.cuda.synchronize()
    wrong, errors = [], []

    def work(q):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(60 if q == 0 else 240):
                    got = net.predict(X[q])
                    if not torch.equal(got, want[q]):
                        wrong.append(q)
        except Exception as e:  # noqa: BLE001 (a thread's failure is the test's)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not wrong, (errors, len(wrong))


def test_buffers_by_tiles_of_rows(cuda_device, monkeypatch):
    """Passes whose numbers of GEMM tiles differ write no buffer in common; there is one pair per such number."""
    import torch

    from elanfmt_gb300.surrogate import MLP

    net = MLP([128, 256, 256, 128], seed=4)
    X = torch.randn(400, 128, device="cuda").to(torch.bfloat16)
    inner, used = net._forward, {}

    def spy(X_, H, P, Y, M):
        used.setdefault(-(-M // 128), set()).add(tuple(H))
        inner(X_, H, P, Y, M)

    monkeypatch.setattr(net, "_forward", spy)
    for n in (400, 1, 100, 128, 129, 256, 300, 384, 400):
        net.predict(X[:n])
    assert sorted(used) == [1, 2, 3, 4] and all(len(v) == 1 for v in used.values())
    buffers = [p for v in used.values() for h in v for p in h]
    assert len(set(buffers)) == len(buffers) == 8
