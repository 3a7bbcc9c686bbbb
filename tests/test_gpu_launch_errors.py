"""A launch that the runtime refuses is an error of its own call alone: the
calls after it do not find it again."""
import ctypes as C

import numpy as np
import pytest

from csrst_b200 import Simulation
from csrst_b200.workloads import make_bunch, workload

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_reported_once(gpu_lib):
    import torch
    x = torch.ones(4, device="cuda")
    p = C.c_void_p(x.data_ptr())
    # 65536 slabs of 256 rows: one more than a grid's second extent may be, so nothing runs
    assert gpu_lib.csrst_nn_colsum(p, 65536 * 256, 1, p, p, 0, None) == -2
    cfg, spec = workload("small-0")
    s = Simulation(cfg)
    s.load(*make_bunch(spec))            # ends by asking for the runtime's last error
    s.step(2)
    assert np.isfinite(s.particles()[0]).all()
    assert bool((x == 1).all())
