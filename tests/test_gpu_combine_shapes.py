"""ewf_mlp_combine over input counts (register and general form), time lengths and alignments: the same
sums in the same order as a serial fp32 loop, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from elanfmt_gb300.solver import load_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nin", [1, 2, 3, 4, 5, 8, 10, 13, 16, 17, 40])
@pytest.mark.parametrize("T,shift", [(1, 0), (3, 0), (4, 0), (4, 1), (127, 0), (512, 0), (516, 2), (1030, 0)])
def test_combine_sums(cuda_device, nin, T, shift):
    import torch

    lib = load_library()
    M, nout = 3, 18
    rng = np.random.default_rng(nin * 7 + T)
    R = rng.normal(size=(M, nout, nin)).astype(np.float32)
    G = rng.normal(size=(M, nin, T)).astype(np.float32)
    want = np.zeros((M, nout, T), np.float32)
    for f in range(nin):  # fp32 product, fp32 sum, input by input
        want += R[:, :, f, None] * G[:, None, f]
    Rg = torch.from_numpy(R).cuda()
    Gg = torch.empty(M * nin * T + shift, device="cuda")[shift:]
    out = torch.full((M * nout * T + shift + 8,), 7.0, device="cuda")
    Gg.copy_(torch.from_numpy(G).reshape(-1))
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.ewf_mlp_combine(p(Rg), p(Gg), p(out[shift:]), M, nout, nin, T, None) == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[shift:shift + want.size].reshape(want.shape), want)
    assert (got[:shift] == 7.0).all() and (got[shift + want.size:] == 7.0).all()
