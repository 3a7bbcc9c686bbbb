"""One network's wakes from several streams, and from several threads on one
stream, at the same time: each is the wake of its own bunches, bit for bit."""
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 70])
def test_wakes_on_several_streams_and_threads(gpu_lib, n):
    import torch
    from csrst_b200 import surrogate
    net = surrogate.FNO(layers=2, seed=5)
    g = torch.Generator().manual_seed(n)
    Xs = [torch.randn(n, 256, 64, generator=g).to(torch.bfloat16).cuda() for _ in range(3)]
    ref = [net.predict(x) for x in Xs]
    torch.cuda.synchronize()
    assert not torch.equal(ref[0], ref[1])
    streams = [torch.cuda.Stream() for _ in Xs]
    got = []
    for _ in range(8):
        for x, s in zip(Xs, streams):
            with torch.cuda.stream(s):
                got.append(net.predict(x))
    torch.cuda.synchronize()
    for k, y in enumerate(got):
        assert torch.equal(y, ref[k % 3])
    res = [None] * 3

    def work(k):
        res[k] = [net.predict(Xs[k]) for _ in range(8)]

    ts = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    net.check()
    for k in range(3):
        for y in res[k]:
            assert torch.equal(y, ref[k])
