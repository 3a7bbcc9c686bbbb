"""The GEMM epilogue's row and column stores, its two ways of reading the
column bias and its prepared divisions, at the edges of tiles and pieces, against an
FP64 product of the same BF16 values.

Bounds: the FP32 accumulation of K <= 192 products and the activation's
approximation (1.5e-7 of its argument's scale) stay within 1e-4 of the largest value; a
BF16 copy adds half a unit of its last place, 2^-8 of each value."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,batch", [(1, 16, 1), (32, 32, 1), (33, 128, 7), (127, 80, 3), (128, 384, 5), (500, 96, 3)])
@pytest.mark.parametrize("bias_off", [0, 1, None])
@pytest.mark.parametrize("row_bias", [False, True])
def test_row_and_column_stores(gpu_lib, M, N, batch, bias_off, row_bias):
    import torch
    from csrst_b200.tensor import check_errors, gemm
    K, ld, alpha = 192, N + 8, 0.75
    g = torch.Generator().manual_seed(M * 1000 + N)
    a = torch.randn(batch, M, K, generator=g).to(torch.bfloat16)
    b = torch.randn(batch, N, K, generator=g).to(torch.bfloat16)
    bias, bm = torch.randn(N + 4, generator=g), torch.randn(M, generator=g)
    bias_d, bm_d = bias.cuda(), bm.cuda()
    pre = torch.full((batch, M, ld), 9.0, device="cuda")
    o32 = torch.full((batch, M, ld), 9.0, device="cuda")
    o16 = torch.full((batch, M, ld), 9.0, dtype=torch.bfloat16, device="cuda")
    Mp = (M + 7) // 8 * 8
    o16t = torch.full((batch, N, Mp), 9.0, dtype=torch.bfloat16, device="cuda")
    gemm(a.cuda(), b.cuda(), M, N, K, batch=batch, stride_a=M * K, stride_b=N * K, alpha=alpha,
         bias=None if bias_off is None else bias_d[bias_off:], bias_m=bm_d if row_bias else None,
         pre=pre, out32=o32, out16=o16, act=1, omap=dict(md=1, nd=1, sm0=ld, sm1=0, sn0=1, sn1=0), sb=M * ld,
         out16t=o16t, tmap=dict(md=1, nd=1, sm0=1, sm1=0, sn0=Mp, sn1=0), tb=N * Mp)
    torch.cuda.synchronize()
    check_errors()
    h = alpha * (a.double() @ b.double().transpose(1, 2))
    if bias_off is not None:
        h = h + bias[bias_off:bias_off + N].double()
    if row_bias:
        h = h + bm.double()[:, None]
    act = 0.5 * h * (1 + torch.erf(h / math.sqrt(2)))
    tol = 1e-4 * float(h.abs().max())
    assert float((pre.cpu()[..., :N].double() - h).abs().max()) <= tol
    assert float((o32.cpu()[..., :N].double() - act).abs().max()) <= tol
    lim = tol + act.abs() * 2.0 ** -8
    assert bool(((o16.cpu()[..., :N].double() - act).abs() <= lim).all())
    assert bool(((o16t.cpu()[..., :M].double().transpose(1, 2) - act).abs() <= lim).all())
    # one value, one rounding: the BF16 copies are the FP32 output's, and the padding is untouched
    assert torch.equal(o16.cpu()[..., :N], o32.cpu()[..., :N].to(torch.bfloat16))
    assert torch.equal(o16t.cpu()[..., :M].transpose(1, 2), o16.cpu()[..., :N])
    assert bool((pre[..., N:] == 9).all() and (o32[..., N:] == 9).all() and (o16[..., N:] == 9).all())
    assert bool((o16t[..., M:] == 9).all())


@pytest.mark.parametrize("M,N,batch", [(32, 32, 1), (33, 48, 2), (128, 128, 3), (250, 160, 2)])
@pytest.mark.parametrize("columns", [False, True])
def test_adding_to_the_output(gpu_lib, M, N, batch, columns):
    """accumulate through row and column runs and the ragged edge, with a BF16 copy of the
    product alone: the FP32 output is the one addition of the old value, exactly."""
    import torch
    from csrst_b200.tensor import check_errors, gemm
    K, Mp = 64, (M + 7) // 8 * 8
    g = torch.Generator().manual_seed(M + N)
    a = torch.randn(batch, M, K, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(batch, N, K, generator=g).to(torch.bfloat16).cuda()
    shape = (batch, N, Mp) if columns else (batch, M, N)
    old = torch.randn(shape, generator=g).cuda()
    omap = dict(md=1, nd=1, sm0=1, sm1=0, sn0=Mp, sn1=0) if columns else None
    sb = shape[1] * shape[2]
    once, twice = torch.zeros(shape, device="cuda"), old.clone()
    o16 = torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
    kw = dict(batch=batch, stride_a=M * K, stride_b=N * K, omap=omap, sb=sb)
    gemm(a, b, M, N, K, out32=once, **kw)
    gemm(a, b, M, N, K, out32=twice, out16=o16, accumulate=True, **kw)
    torch.cuda.synchronize()
    check_errors()
    r = a.double() @ b.double().transpose(1, 2)
    got = once.transpose(1, 2)[:, :M] if columns else once
    assert float((got.double() - r).abs().max()) <= 1e-4 * float(r.abs().max())
    assert torch.equal(twice, old + once)
    assert torch.equal(o16, once.to(torch.bfloat16))
