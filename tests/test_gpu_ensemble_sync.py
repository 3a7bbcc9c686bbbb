"""Ensemble.sync reads all members' errors at once, and the device-side wake read carries
the member's window origin and mean."""
import ctypes as C

import numpy as np
import pytest

from csrst_b200 import Ensemble, Simulation
from csrst_b200.workloads import make_bunch, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [1, 3, 130])
def test_sync_and_wake_of_members(gpu_lib, members):
    import torch
    cfg, spec = workload("small-0")
    sims = []
    for k in range(members):
        s = Simulation(cfg, fp32=True)
        s.load(*make_bunch(spec))
        sims.append(s)
    ens = Ensemble(sims)
    ens.step(2)
    ens.sync()
    s = sims[-1]
    n = s.window()[0][2] - 4
    out, meta = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (n, 4))
    assert gpu_lib.csrst_diag_wake_async(s.h, C.c_void_p(out.data_ptr()), n, C.c_void_p(meta.data_ptr())) == 0
    s.sync()
    assert np.array_equal(out.cpu().numpy(), s.wake(), equal_nan=True)
    m = meta.cpu().numpy()
    assert np.array_equal(m[:2], s.window()[1]) and np.array_equal(m[2:], s.moments()[:2])
    bad = C.c_int(7)
    assert gpu_lib.csrst_ensemble_sync(ens._e, C.byref(bad)) == 0 and bad.value == -1
    ens.close()
    for s in sims:
        s.close()
