"""Inference with one network from several streams and threads, at the host (no
GPU needed: the library's forward pass is stood in for): passes on two streams use
buffers of their own, passes of two threads on one stream go out one after the other."""
import ctypes as C
import threading
import time
import types

import pytest
import torch

from csrst_b200 import surrogate


class Library:
    """Records each forward pass's spectra buffer, its stream and whether another pass was going out on them."""

    def __init__(self):
        self.passes, self.busy, self.overlaps = [], set(), 0

    def csrst_fno_refresh(self, *a):
        return 0

    def csrst_fno_forward(self, net, X, out, err, stream):
        at = (net._obj.U16, net._obj.V16)
        self.passes.append((stream.value, net._obj.U16, net._obj.batch))
        self.overlaps += at[0] in self.busy
        self.busy.add(at[0])
        time.sleep(0.02)
        self.busy.discard(at[0])
        return 0


@pytest.fixture
def net(monkeypatch):
    here = threading.local()
    L = Library()
    monkeypatch.setattr(surrogate, "lib", lambda: L)
    monkeypatch.setattr(surrogate, "_stream", lambda: C.c_void_p(getattr(here, "stream", 0)))
    net = surrogate.FNO(width=64, modes=32, layers=2, nout=16, seed=1, device="cpu")
    return types.SimpleNamespace(net=net, L=L, here=here)


def X(n):
    return torch.zeros(n, surrogate.NBINS, surrogate.NFEAT, dtype=torch.bfloat16)


def test_streams_have_buffers_of_their_own(net):
    for stream in (0, 0x70, 0x80, 0x70):
        net.here.stream = stream
        net.net.predict(X(3))
    at = {}
    for stream, u, _ in net.L.passes:
        at.setdefault(stream, set()).add(u)
    assert [len(v) for v in at.values()] == [1, 1, 1]     # kept from call to call
    assert len(set.union(*at.values())) == 3


def test_chunks_on_one_stream(net):
    out = net.net.predict(X(7), chunk=3)
    assert out.shape == (7, surrogate.NBINS, 16)
    assert [b for _, _, b in net.L.passes] == [3, 3, 1]
    assert net.L.passes[0][1] == net.L.passes[1][1]


def test_threads_on_one_stream_take_turns(net):
    ts = [threading.Thread(target=lambda: [net.net.predict(X(2)) for _ in range(4)]) for _ in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(net.L.passes) == 16 and net.L.overlaps == 0


def test_training_keeps_one_set(net):
    a = net.net._buf(2, True)
    net.here.stream = 0x70
    assert net.net._buf(2, True) is a and net.net._bufs[(2, True)] is a
