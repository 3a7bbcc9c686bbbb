"""Inference with many different numbers of bunches keeps a few sets of buffers,
each large enough for what runs on it (host only; the library's forward pass is
stood in for as in test_fno_concurrent)."""
import torch

from csrst_b200 import surrogate
from test_fno_concurrent import X, net  # noqa: F401


def bytes_kept(n):
    return sum(t.numel() * t.element_size() for bf in n._bufs.values() for v in vars(bf).values()
               for t in (v if isinstance(v, list) else [v]) if torch.is_tensor(t))


def test_many_batch_sizes(net, monkeypatch):  # noqa: F811
    monkeypatch.setattr("time.sleep", lambda s: None)
    sizes = {}
    real = net.L.csrst_fno_forward

    def forward(ref, *a):
        f = ref._obj
        (bf,) = [b for b in net.net._bufs.values() if b.U16.data_ptr() == f.U16]
        B, w, m = f.batch, f.width, f.modes
        assert bf.U16.numel() >= m * B * 2 * w and bf.Z16.numel() >= m * B * 2 * w
        assert bf.Zp16.numel() >= B * w * 2 * m and bf.A1_16.numel() >= B * surrogate.NBINS * w
        assert all(v.numel() >= B * surrogate.NBINS * w for v in bf.V16)
        sizes[B] = f.U16
        return real(ref, *a)

    monkeypatch.setattr(net.L, "csrst_fno_forward", forward, raising=False)
    x = X(70)
    for n in range(1, 71):
        assert net.net.predict(x[:n]).shape[0] == n
    assert len(sizes) == 70
    assert len(net.net._bufs) <= 8                       # 1, 2, 4 ... 128
    one = surrogate._Buffers(net.net, 128, False)
    assert bytes_kept(net.net) <= 2 * bytes_kept(type("N", (), {"_bufs": {0: one}}))
