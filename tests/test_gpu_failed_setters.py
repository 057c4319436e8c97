"""A setter that fails leaves a handle that runs: without receivers, and with those that are set next."""
import numpy as np
import pytest

from elanfmt_gb300 import fields as F
from elanfmt_gb300 import inputs as I
from elanfmt_gb300.solver import EwfError, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 20, 12), (80, 76, 70)])  # one and two cells per thread
def test_receivers_whose_traces_do_not_fit(cuda_device, shape):
    nt = 2_000_000
    m = I.random_small(F.MODEL_ISO, *shape, nt=40, seed=4)
    m.nt, m.stf = nt, np.concatenate([m.stf, np.zeros(nt - len(m.stf))])
    few = np.array([(5, 6, 1, F.F_VX), (7, 3, 4, F.F_VZ)], np.int32)
    many = np.tile(few, (150000, 1))  # 4.8 TB of samples
    m.receivers = few
    with Solver.from_model(m, check_finite=False) as s:
        s.run(70)
        with pytest.raises(EwfError) as e:
            s.set_receivers(many)
        assert e.value.status == -3
        s.run(70)                                   # nothing is recorded
        s.set_receivers(few)
        s.run(70)
        tr, vz = s.seismograms(), s.field(F.F_VZ)
    with Solver.from_model(m, check_finite=False) as s:
        s.run(210)
        ref = s.seismograms()
        np.testing.assert_array_equal(vz, s.field(F.F_VZ))
    assert not tr[:, :140].any()
    np.testing.assert_array_equal(tr[:, 140:210], ref[:, 140:210])
    assert np.abs(ref).max() > 0
