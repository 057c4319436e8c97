"""The device band-pass on many, short and few-section traces, where a thread per trace is the faster form: the
host path's bits, and the FP64 pipe kept busy."""
import numpy as np
import pytest

from elanfmt_gb300 import postproc as P

pytestmark = pytest.mark.gpu


def _sections(n, seed):
    rng = np.random.default_rng(seed)
    r, th = rng.uniform(0.3, 0.95, n), rng.uniform(0, np.pi, n)
    return np.column_stack([rng.normal(size=(n, 3)), np.full(n, 1.7), -2 * 1.7 * r * np.cos(th), 1.7 * r * r])


@pytest.mark.parametrize("sections", [1, 3, 4, 5, 9, 16])
@pytest.mark.parametrize("traces,samples", [(1, 1), (2, 15), (65, 3), (64, 17), (3001, 40), (9727, 33), (20001, 21)])
def test_many_or_short_traces(cuda_device, sections, traces, samples):
    import torch

    sos = _sections(sections, sections + traces)
    x = np.random.default_rng(traces).normal(size=(traces, samples))
    t = torch.from_numpy(x.copy()).cuda()
    P.sosfilt_device(sos, t)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(t.cpu().numpy(), P.sosfilt(sos, x))


@pytest.mark.parametrize("sections,traces,samples,bound_ms", [
    # an FP64 instruction of a warp takes an SM 19 cycles, 9 of them a section and sample: 1.2 and 1.5 ms at 1.92 GHz; twice that
    (4, 1000000, 16, 2.4), (5, 400000, 40, 3.0)])
def test_many_traces_keep_the_pipe_busy(cuda_device, sections, traces, samples, bound_ms):
    import torch

    sos = _sections(sections, 7)
    x = torch.randn(traces, samples, dtype=torch.float64, device="cuda")
    times = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        P.sosfilt_device(sos, x)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    assert min(times) < bound_ms, times
