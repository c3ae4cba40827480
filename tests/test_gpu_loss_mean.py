"""The one-CTA mean over the row losses (ulm_loss_mean) at the edges of its 1024-thread stride."""
import ctypes as C

import pytest
import torch

import _native as N

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
