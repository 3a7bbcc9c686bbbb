"""The surrogate's element-wise kernels at the edges of their forms: tiles and
remainders of the transposes, packed and unpacked spectral weights, column sums
of one and more slabs, casts and the optimiser off a multiple of four, misaligned
pointers.

Data movement is exact.  Sums: each column against the same order of FP32 additions in
numpy, exactly.  The optimiser: within 2^-20 of FP64 (four FP32 roundings of the moments, a
square root and two quotients)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ptr(t, off=0):
    return C.c_void_p(t.data_ptr() + off * t.element_size())


@pytest.mark.parametrize("batch,rows,cols,pad", [(1, 64, 64, 0), (3, 128, 192, 8), (2, 64, 64, 3), (1, 63, 65, 1),
                                                 (2, 32, 128, 0), (1, 96, 129, 4), (1, 32, 7, 0), (1, 1, 1, 0)])
@pytest.mark.parametrize("off", [0, 1])
def test_transposes(gpu_lib, batch, rows, cols, pad, off):
    import torch
    for dt, f in ((torch.int16, gpu_lib.csrst_nn_transpose_bf16), (torch.int32, gpu_lib.csrst_nn_transpose_b32)):
        src = torch.arange(off + batch * rows * cols, device="cuda").to(dt)
        dst = torch.full((off + batch * cols * (rows + pad),), -7, dtype=dt, device="cuda")
        assert f(ptr(src, off), ptr(dst, off), batch, rows, cols, rows + pad, None) == 0
        torch.cuda.synchronize()
        got = dst[off:].view(batch, cols, rows + pad)
        assert torch.equal(got[..., :rows], src[off:].view(batch, rows, cols).transpose(1, 2))
        assert bool((got[..., rows:] == -7).all()) and bool((dst[:off] == -7).all())


@pytest.mark.parametrize("modes,ch", [(1, 1), (3, 31), (2, 33), (2, 64)])
@pytest.mark.parametrize("off", [0, 1])
def test_spectral_pack_and_unpack(gpu_lib, modes, ch, off):
    import torch
    g = torch.Generator().manual_seed(ch)
    wr, wi = torch.randn(modes, ch, ch, generator=g), torch.randn(modes, ch, ch, generator=g)
    wrd, wid = wr.cuda(), wi.cuda()
    mk = torch.zeros(off + modes * 4 * ch * ch, dtype=torch.bfloat16, device="cuda")
    mkt = torch.zeros_like(mk)
    assert gpu_lib.csrst_nn_spectral_pack(ptr(wrd), ptr(wid), modes, ch, ptr(mk, off), ptr(mkt, off), None) == 0
    ref = torch.zeros(modes, ch, 2, ch, 2)      # [k][o][p][c][q]
    r, i = wr.transpose(1, 2), wi.transpose(1, 2)
    ref[:, :, 0, :, 0], ref[:, :, 0, :, 1], ref[:, :, 1, :, 0], ref[:, :, 1, :, 1] = r, -i, i, r
    ref = ref.reshape(modes, 2 * ch, 2 * ch).to(torch.bfloat16)
    assert torch.equal(mk[off:].view_as(ref).cpu(), ref)
    assert torch.equal(mkt[off:].view_as(ref).cpu(), ref.transpose(1, 2))
    d = torch.randn(modes, 2 * ch, 2 * ch, generator=g)
    dd, dwr, dwi = d.cuda(), torch.zeros_like(wrd), torch.zeros_like(wid)
    assert gpu_lib.csrst_nn_spectral_unpack(ptr(dd), modes, ch, ptr(dwr), ptr(dwi), None) == 0
    v = d.view(modes, ch, 2, ch, 2)
    assert torch.equal(dwr.cpu(), (v[:, :, 0, :, 0] + v[:, :, 1, :, 1]).transpose(1, 2))
    assert torch.equal(dwi.cpu(), (v[:, :, 1, :, 0] - v[:, :, 0, :, 1]).transpose(1, 2))


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (256, 64), (257, 65), (800, 32)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_column_sums_in_order(gpu_lib, rows, cols, accumulate):
    import torch
    x = np.random.default_rng(rows).standard_normal((rows, cols)).astype(np.float32)
    slabs = (rows + 255) // 256
    xd, part = torch.from_numpy(x).cuda(), torch.empty(slabs * cols, device="cuda")
    out = torch.full((cols,), 0.5, device="cuda")
    assert gpu_lib.csrst_nn_colsum(ptr(xd), rows, cols, ptr(part), ptr(out), accumulate, None) == 0
    total = np.zeros(cols, dtype=np.float32)
    for k in range(slabs):
        s = np.zeros(cols, dtype=np.float32)
        for r in x[256 * k:256 * k + 256]:
            s = s + r
        total = total + s
    assert np.array_equal(out.cpu().numpy(), total + np.float32(0.5) if accumulate else total)


@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (4096, 0), (4096, 1), (1 << 20, 0)])
def test_cast_loss_and_adam(gpu_lib, n, off):
    import torch
    g = torch.Generator().manual_seed(n)
    w, gr, m = (torch.randn(n + off, generator=g) for _ in range(3))
    v = torch.rand(n + off, generator=g)
    wd, gd, md, vd = w.cuda(), gr.cuda(), m.cuda(), v.cuda()
    y = torch.zeros(n + off, dtype=torch.bfloat16, device="cuda")
    assert gpu_lib.csrst_nn_cast_bf16(ptr(wd, off), ptr(y, off), n, None) == 0
    assert torch.equal(y[off:].cpu(), w[off:].to(torch.bfloat16))
    part, loss = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (256, 1))
    grad = torch.zeros(n * 2, device="cuda")
    assert gpu_lib.csrst_nn_mse(ptr(wd, off), ptr(gd, off), None, n, ptr(grad), 1, 2, 0, ptr(part), ptr(loss), None) == 0
    e = (w[off:] - gr[off:])
    assert float(loss) == pytest.approx(float((e.double() ** 2).mean()), rel=1e-12)
    assert torch.allclose(grad.cpu()[::2], 2 * e / n, rtol=2.0 ** -22, atol=0) and not bool(grad.cpu()[1::2].any())
    coef = torch.tensor([1e-2, 0.1, 0.2], device="cuda")
    assert gpu_lib.csrst_nn_adam(ptr(wd, off), ptr(gd, off), ptr(md, off), ptr(vd, off), n, ptr(coef), 0.9, 0.999,
                                 1e-8, None) == 0
    lr, c1, c2 = (float(c) for c in coef.double())
    b1, b2, eps = (float(np.float32(c)) for c in (0.9, 0.999, 1e-8))
    m2 = b1 * m.double() + float(np.float32(1) - np.float32(0.9)) * gr.double()
    v2 = b2 * v.double() + float(np.float32(1) - np.float32(0.999)) * gr.double() ** 2
    step = lr * (m2 / c1) / ((v2 / c2).sqrt() + eps)
    tol = 2.0 ** -20
    assert bool(((md.cpu().double() - m2).abs() <= tol * (m.abs() + gr.abs()))[off:].all())
    assert bool(((vd.cpu().double() - v2).abs() <= tol * v2)[off:].all())
    lim = tol * (w.abs() + step.abs() + lr * (m.abs() + gr.abs()) / c1 / (v2 / c2).sqrt())
    assert bool(((wd.cpu().double() - (w.double() - step)).abs() <= lim)[off:].all())
    assert torch.equal(wd[:off].cpu(), w[:off])
