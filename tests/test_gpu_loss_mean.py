"""The one-CTA mean over the row losses (ulm_loss_mean) at the edges of its 1024-thread stride."""
import ctypes as C

import pytest
import torch

import _native as N
import ulm_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('rows', [1, 31, 1023, 1024, 1025, 4097, 40001])
@pytest.mark.parametrize('form', ['count', 'all ignored', 'host', 'device'])
def test_loss_mean_matches_float64(rows, form):
    g = torch.Generator().manual_seed(rows)
    target = torch.randint(1, 50, (rows,), generator=g)
    target[torch.rand(rows, generator=g) < 0.3] = 0
    if form == 'all ignored':
        target.zero_()
    losses = torch.rand(rows, generator=g) * (target != 0)
    lc, tc, out = losses.cuda(), target.cuda(), torch.empty(2, device='cuda')
    dev = torch.full((1,), 777.0, device='cuda') if form == 'device' else None
    N.check(N.lib().ulm_loss_mean(lc.data_ptr(), tc.data_ptr(), rows, 0, dev.data_ptr() if dev is not None else None,
                                  123.5 if form == 'host' else 0.0, out[0:].data_ptr(), out[1:].data_ptr(),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)), 'loss_mean')
    n = {'device': 777.0, 'host': 123.5}.get(form, max(1, int((target != 0).sum())))
    # fp32 summation of non-negative terms in a tree of depth log2: a few ulp
    want = float(losses.double().sum()) / n
    assert abs(float(out[0]) - want) <= 2e-6 * max(want, 1e-30) + 1e-12
    assert abs(float(out[1]) * n - 1.0) <= 2e-7


@pytest.mark.parametrize('rows', [1025, 32768, 40001, 300007])
def test_loss_mean_is_rounded_once(rows):
    losses = torch.rand(rows, generator=torch.Generator().manual_seed(rows)) * 12
    lc, tc, out = losses.cuda(), torch.ones(rows, dtype=torch.long).cuda(), torch.empty(2, device='cuda')
    N.check(N.lib().ulm_loss_mean(lc.data_ptr(), tc.data_ptr(), rows, 0, None, 0.0, out[0:].data_ptr(), out[1:].data_ptr(),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)), 'loss_mean')
    # an fp64 sum is exact to 2^-53 * rows: what remains is the one rounding to fp32
    want = float(losses.double().sum()) / rows
    assert abs(float(out[0]) - want) <= 2.0 ** -24 * want * (1 + 1e-6)


@pytest.mark.parametrize('kept', [True, False])
@pytest.mark.parametrize('denominator', [0, -4.0, float('nan'), 7, torch.tensor(5), torch.tensor([5.0]), torch.tensor([[2.0, 4.0]])])
def test_cross_entropy_divides_by_the_denominator_it_is_given(denominator, kept, monkeypatch):
    monkeypatch.setattr(ulm_ops, 'KEEP_LOGITS_BYTES', ulm_ops.KEEP_LOGITS_BYTES if kept else 0)
    g = torch.Generator(device='cuda').manual_seed(1)
    h, w = (torch.randn(s, 64, generator=g, device='cuda').half().requires_grad_() for s in (40, 128))
    t = torch.randint(1, 128, (40,), generator=g, device='cuda')
    total = ulm_ops.chunked_cross_entropy(h, w, t, denominator=1.0)
    got = ulm_ops.chunked_cross_entropy(h, w, t, denominator=denominator)
    want = total / (denominator.cuda() if torch.is_tensor(denominator) else denominator)
    assert got.shape == want.shape and torch.allclose(got, want, rtol=1e-6, equal_nan=True)
    if got.numel() == 1 and torch.isfinite(got).all():
        # the logits' gradients and what is summed from them are rounded to fp16 (half an ulp: 2^-11 of a value at most), in
        # each of the two: 4 such errors, as 2-norms because single elements cancel
        a, b = torch.autograd.grad(got.sum(), h)[0].double(), torch.autograd.grad(total, h)[0].double() / float(denominator)
        assert float((a - b).norm()) <= 4 * 2.0 ** -11 * float(b.norm())
