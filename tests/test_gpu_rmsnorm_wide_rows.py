"""Residual add + RMSNorm backward for rows of 769 to 1024 elements (four warps a row, x and dy of the next row requested ahead): ragged
widths, row counts around a CTA's three rows and around one pass of the full grid (296 CTAs, 888 rows), with and without a gradient at
the sum."""
import pytest
import torch


@pytest.mark.parametrize('rows,parts', [(0, 1), (1, 1), (3, 1), (4, 2), (512, 171), (885, 295), (886, 296), (888, 296), (100000, 296)])
def test_partial_rows_cover_a_cta_per_three_rows(rows, parts):
    """The grid is capped by the partial rows: with fewer, rows wait for a CTA while SMs have none."""
    import _native
    assert _native.lib().ulm_rmsnorm_bwd_partial_rows(rows) == parts


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
@pytest.mark.parametrize('rows,d', [(1, 1024), (2, 772), (3, 900), (4, 1020), (887, 1024), (889, 772), (1777, 1024), (2665, 1000)])
@pytest.mark.parametrize('with_sum', [True, False])
def test_add_norm_backward(dtype, rows, d, with_sum):
    """Against fp64.  fp32 throughout: sums of at most 1024 terms (1e-6 relative) for dx, of `rows` terms for dw; the branch's gradient is
    dx rounded once (2^-9 in bf16, 2^-12 in fp16)."""
    import ulm_ops
    g = torch.Generator(device='cuda').manual_seed(rows + d)
    x = torch.randn((rows, d), generator=g, device='cuda').requires_grad_(True)
    br = torch.randn((rows, d), generator=g, device='cuda').to(dtype).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(d, generator=g, device='cuda')).requires_grad_(True)
    gy = torch.randn((rows, d), generator=g, device='cuda').to(dtype)
    gx = torch.randn((rows, d), generator=g, device='cuda')
    x_new, y = ulm_ops.add_rms_norm(x, br, w, 1e-6)
    outs, grads = ([x_new, y], [gx, gy]) if with_sum else ([y], [gy])
    dx, db, dw = torch.autograd.grad(outs, [x, br, w], grads)
    s, wd, gyd = (x + br).detach().double(), w.detach().double(), gy.double()
    inv = (s.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    want = inv * (gyd * wd - s * inv * inv * (gyd * wd * s).mean(-1, keepdim=True)) + (gx.double() if with_sum else 0)
    torch.testing.assert_close(dx.double(), want, rtol=1e-4, atol=1e-5)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    torch.testing.assert_close(db.double(), want, rtol=eps, atol=1e-5)
    dw_want = (gyd * s * inv).sum(0)
    assert float((dw.double() - dw_want).norm() / dw_want.norm()) < 1e-5
