"""Networks that have trained are copied and unpickled on a host without a GPU
(torch.load(..., map_location="cpu") of one trained elsewhere): the parameters
are all there, and the second stream of a training step is made when a step needs it."""
import copy
import io
import types

import torch

from csrst_b200 import surrogate


def trained(monkeypatch):
    """A network on the host with the buffers of a training batch (no launches)."""
    monkeypatch.setattr(surrogate, "lib", lambda: types.SimpleNamespace(csrst_fno_refresh=lambda *a: 0))
    monkeypatch.setattr(surrogate, "_stream", lambda: None)
    net = surrogate.FNO(width=64, modes=32, layers=1, nout=16, seed=3, device="cpu")
    bf = surrogate._Buffers.__new__(surrogate._Buffers)
    vars(bf).update(train=True, V16=[torch.ones(4)], loss=torch.ones(1, dtype=torch.float64))
    net._bufs[(64, True)] = bf
    return net


def test_copies_without_a_gpu(monkeypatch):
    net = trained(monkeypatch)
    f = io.BytesIO()
    torch.save(net, f)
    f.seek(0)
    for other in (copy.deepcopy(net), torch.load(f, map_location="cpu", weights_only=False)):
        assert other.w is not net.w and torch.equal(other.w, net.w)
        assert set(other.params()) == set(net.params())
        assert torch.equal(other._bufs[(64, True)].loss, net._bufs[(64, True)].loss)


def test_buffers_saved_with_no_stream(monkeypatch):
    """Whatever of a stream a buffer set holds stays out of its copies."""
    bf = trained(monkeypatch)._bufs[(64, True)]
    bf.side = object()                     # (stands for a torch.cuda.Stream)
    other = copy.deepcopy(bf)
    assert other.side is None and "side" not in vars(other)
