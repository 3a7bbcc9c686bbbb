"""A thread's first CUDA work may be a call of this library: a product, a
network's wakes and a batch of simulations made in a fresh thread."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_thread(f):
    out = []

    def run():
        try:
            out.append(f())
        except BaseException as e:      # noqa: BLE001 (handed to the caller)
            out.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if isinstance(out[0], BaseException):
        raise out[0]
    return out[0]


def test_products_in_a_fresh_thread(gpu_lib):
    import torch
    from csrst_b200 import surrogate
    from csrst_b200.tensor import gemm
    A = torch.randn(200, 128, device="cuda").to(torch.bfloat16)
    B = torch.randn(64, 128, device="cuda").to(torch.bfloat16)
    a, b = torch.empty(200, 64, device="cuda"), torch.empty(200, 64, device="cuda")
    net = surrogate.FNO(layers=1, seed=2)
    X = torch.randn(5, 256, 64, device="cuda").to(torch.bfloat16)
    gemm(A, B, 200, 64, 128, out32=a)
    ref = net.predict(X)
    torch.cuda.synchronize()
    in_thread(lambda: gemm(A, B, 200, 64, 128, out32=b))
    wake = in_thread(lambda: net.predict(X))
    torch.cuda.synchronize()
    assert torch.equal(a, b) and torch.equal(ref, wake)


@pytest.mark.parametrize("fp32", [False, True])
def test_steps_in_a_fresh_thread(gpu_lib, fp32):
    from csrst_b200 import Simulation
    from csrst_b200.pic import Ensemble
    from csrst_b200.workloads import make_bunch, workload

    def sims():
        out = []
        for name in ("small-0", "small-1"):
            cfg, spec = workload(name)
            s = Simulation(cfg, fp32=fp32)
            s.load(*make_bunch(spec))
            out.append(s)
        return out

    a, b, c = sims(), sims(), sims()
    ea, eb = Ensemble(a), in_thread(lambda: Ensemble(b))
    ea.step(4)
    ea.sync()
    in_thread(lambda: eb.step(4))
    in_thread(lambda: eb.sync())
    for s in c:
        in_thread(lambda: s.step(4))
    for x, y, z in zip(a, b, c):
        for p, q, r in zip(x.particles(), y.particles(), z.particles()):
            assert np.array_equal(p, q) and np.array_equal(p, r)
    ea.close()
    eb.close()
