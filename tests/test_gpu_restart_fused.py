"""A restored handle steps as a loaded one does: through the fused field sweep
(the sweep alone has staging waits, so their stuck-wait hook tells which path
ran) and, bit for bit, to the results of the run that was not interrupted, singly,
in a handle that held another bunch before, and as a member of an ensemble."""
import numpy as np
import pytest

from csrst_b200 import CsrstError, Simulation
from csrst_b200.pic import Ensemble
from csrst_b200.workloads import make_bunch, workload
from test_gpu_checkpoint import state

pytestmark = pytest.mark.gpu


def loaded(name, fp32):
    cfg, spec = workload(name)
    s = Simulation(cfg, fp32=fp32)
    s.load(*make_bunch(spec))
    return s


@pytest.mark.parametrize("fp32", [False, True])
def test_restored_run_takes_the_fused_sweep(gpu_lib, tmp_path, fp32):
    cfg, spec = workload("small-1")
    path = str(tmp_path / "run.ckpt")
    a = loaded("small-1", fp32)
    a.step(5)
    a.checkpoint(path)
    stuck, b, c = Simulation(cfg, fp32=fp32), Simulation(cfg, fp32=fp32), Simulation(cfg, fp32=fp32)
    stuck.restore(path)
    try:
        gpu_lib.csrst_set_staging_wait_limit(-200)
        with pytest.raises(CsrstError) as ei:
            stuck.step(3)
            stuck.sync()
        assert ei.value.code == -10
    finally:
        gpu_lib.csrst_set_staging_wait_limit(0)
    x, y, px, py, q = make_bunch(spec)
    c.load(x[: len(x) // 3], y[: len(x) // 3], px[: len(x) // 3], py[: len(x) // 3], q[: len(x) // 3])
    c.step(4)                                   # a captured step of another bunch and window
    b.restore(path)
    c.restore(path)
    member = Simulation(cfg, fp32=fp32)
    member.restore(path)
    for s in (a, b, c):
        s.step(7)
    other = loaded("small-0", fp32)
    ens = Ensemble([member, other])
    ens.step(7)
    ens.sync()
    ref = state(a)
    for s in (b, c, member):
        for u, v in zip(ref, state(s)):
            assert np.array_equal(u, v)
    ens.close()
