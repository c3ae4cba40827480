"""The 16-bit gate's special-function path, over every value a 16-bit input can have and against the divided formula."""
import pytest
import torch

import ulm_ops

pytestmark = pytest.mark.gpu


def _gate(a, b, dy):
    a, b = a.clone().requires_grad_(), b.clone().requires_grad_()
    y = ulm_ops.swiglu(a, b)
    return [y.detach().double(), *(g.double() for g in torch.autograd.grad(y, [a, b], dy))]


@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
def test_every_value(dtype):
    a = torch.arange(-32768, 32768, dtype=torch.int32, device='cuda').to(torch.int16).view(dtype)
    one = torch.ones_like(a)
    y, da, db = _gate(a, one, one)
    x, fi = a.double(), torch.finfo(dtype)
    s = torch.sigmoid(x)
    ok = torch.isfinite(x)

    def bound(want, terms):
        # half an ulp of the result (a fixed one among the subnormals) + the stated relative error of s and u, on the terms
        # that are added; below a = -88 exp(-a) overflows fp32 and what is lost is under 2^-119
        ulp = 2.0 ** torch.floor(torch.log2(want.abs().clamp(min=fi.tiny))) * fi.eps
        return 0.5 * ulp * 1.01 + 2.0 ** -17 * terms + 2.0 ** -119

    u = x * s
    assert bool(((y - u).abs() <= bound(u, u.abs()))[ok].all())
    assert bool(((db - u).abs() <= bound(u, u.abs()))[ok].all())
    want = s * (1 + x * (1 - s))
    # 1 - s has the error of the reciprocal's last place too: 2^-23, 2^-6 of the bound
    assert bool(((da - want).abs() <= bound(want, s * (1 + x.abs() * (1 - s + 2.0 ** -6))))[ok].all())
    nan = torch.isnan(x) | (x == -torch.inf)             # silu(-inf) is -inf / inf in the divided form too
    assert bool(torch.isnan(y[nan]).all()) and float(y[x == torch.inf][0]) == torch.inf


@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
@pytest.mark.parametrize('spread', [0.3, 1.0, 3.0])
def test_error_is_that_of_the_divided_formula(dtype, spread):
    g = torch.Generator(device='cuda').manual_seed(5)
    a, b, dy = ((torch.randn(4096, 2048, generator=g, device='cuda') * m).to(dtype) for m in (spread, 1, 1))
    got = _gate(a, b, dy)
    x, fa, r = a.double(), a.float(), (lambda v: v.to(dtype).float())
    s = torch.sigmoid(x)
    want = (x * s * b.double(), dy.double() * b.double() * s * (1 + x * (1 - s)), dy.double() * x * s)
    d = 1 + torch.exp(-fa)
    sf, u = 1 / d, r(fa / d)
    ref = (r(u * b.float()), r(r(dy.float() * b.float()) * (sf * (1 + fa * (1 - sf)))), r(dy.float() * u))
    for x, e, f in zip(got, want, ref):
        # an error of 2^-19 beside fp16's rounding of rms 2^-11 / sqrt(12) adds up to sqrt(1 + 0.0135^2)
        assert float((x - e).norm()) <= float((f.double() - e).norm()) * (1 + 1e-4)
