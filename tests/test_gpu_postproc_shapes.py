"""The device band-pass over section counts, trace lengths around its tiles and trace counts around
its warps: the host path's bits."""
import numpy as np
import pytest

from elanfmt_gb300 import postproc as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sections", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("samples", [1, 2, 7, 30, 31, 33, 63, 64, 65, 130, 200, 1001])
def test_device_filter_shapes(cuda_device, sections, samples):
    import torch

    rng = np.random.default_rng(sections * 1000 + samples)
    # stable sections of no particular filter: poles inside the unit circle, any zeros
    r, th = rng.uniform(0.3, 0.95, sections), rng.uniform(0, np.pi, sections)
    sos = np.column_stack([rng.normal(size=(sections, 3)), np.full(sections, 1.7), -2 * 1.7 * r * np.cos(th), 1.7 * r * r])
    sos[0, 1] = -0.0 if samples % 2 else sos[0, 1]
    if samples == 200:
        sos[-1, 4:] = 0.0  # no feedback: an infinite sample leaves again
    for traces in (1, 3, 8, 33, 70, 12000):
        if traces == 12000 and samples != 130:  # more traces than run at once
            continue
        x = rng.normal(size=(traces, samples))
        x[rng.random(x.shape) < 0.1] = -0.0
        if traces == 3:
            x[1, samples // 2] = np.inf
        t = torch.from_numpy(x.copy()).cuda()
        P.sosfilt_device(sos, t)
        torch.cuda.synchronize()
        got, want = t.cpu().numpy(), P.sosfilt(sos, x)
        nan = np.isnan(want)
        assert np.array_equal(nan, np.isnan(got))
        assert np.array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64)), (sections, samples, traces)
