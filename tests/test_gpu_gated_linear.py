"""The fused gated projections (ulm_ops.gated_linear) and the gate on column blocks, against two linears and a gate."""
import pytest
import torch

import ulm_ops

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30))


@pytest.mark.parametrize('rows,d,ff', [(1, 64, 8), (31, 128, 344), (257, 128, 2816), (1000, 768, 2048), (5, 64, 12)])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
@pytest.mark.parametrize('form', ['adjacent copies', 'separate copies', 'in place'])
def test_gated_linear_matches_separate_projections(rows, d, ff, dtype, form):
    g = torch.Generator(device='cuda').manual_seed(rows + ff)
    x = torch.randn(rows, d, generator=g, device='cuda').to(dtype).requires_grad_()
    w1, w3 = (torch.nn.Parameter(torch.randn(ff, d, generator=g, device='cuda') * d ** -0.5) for _ in range(2))
    dy = torch.randn(rows, ff, generator=g, device='cuda').to(dtype)
    want = torch.nn.functional.silu(x.double() @ w1.to(dtype).double().t()) * (x.double() @ w3.to(dtype).double().t())
    ref = torch.autograd.grad(want, (x, w1, w3), dy.double())
    copies = ulm_ops.weight_copies([w1, w3], dtype) if form != 'separate copies' else None
    with ulm_ops.weight_cast_scope(copies), torch.autocast('cuda', dtype=dtype), ulm_ops.wgrad_in_place(form == 'in place'):
        if form == 'in place':
            flat = torch.ones(2 * w1.numel(), device='cuda')
            w1.grad, w3.grad = flat[:w1.numel()].view_as(w1), flat[w1.numel():].view_as(w3)
        y = ulm_ops.gated_linear(x, w1, w3)
        if form == 'in place':
            y.backward(dy)
            got = (x.grad, w1.grad - 1, w3.grad - 1)
        else:
            got = torch.autograd.grad(y, (x, w1, w3), dy)
    # a, b, their gradients and the results are each rounded to 16 bits once: a few half ulps, added in quadrature
    tol = 4 * 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert y.dtype == dtype and _rel(y, want) <= tol
    for a, b in zip(got, ref):
        assert a.shape == b.shape and _rel(a, b) <= tol
