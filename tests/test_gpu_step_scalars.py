"""The step's small kernels: token targets and gradient clipping, at the edges of their vectors and blocks."""
import pytest
import torch

import ulm_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,L', [(1, 1), (3, 5), (1, 256), (7, 255), (2, 1024), (30, 1087)])
def test_token_targets(n, L):
    ids = torch.randint(1, 999, (n, L), device='cuda')
    padded = -(-n * L // 1024) * 1024
    flat, target = ulm_ops.token_targets(ids, ids, padded, -7)
    want = torch.full((n, L), -7, device='cuda')
    want[:, :-1] = ids[:, 1:]
    assert torch.equal(flat[:n * L], ids.reshape(-1)) and not flat[n * L:].any()
    assert torch.equal(target[:n * L], want.reshape(-1)) and bool((target[n * L:] == -7).all())


@pytest.mark.parametrize('n', [1, 3, 4, 1023, 1025, 4 * 256 * 16 * 148 + 5])
@pytest.mark.parametrize('scale', [1e-3, 1.0, 37.0])
def test_grad_clip(n, scale):
    g = torch.randn(n, generator=torch.Generator().manual_seed(n)).cuda()
    g *= scale / g.norm()
    want = g.clone()
    sumsq = torch.stack([(g.double() ** 2).sum().float(), g.new_zeros(())])
    norm = ulm_ops.grad_clip_(g, sumsq, 1.0)
    factor = torch.clamp(1.0 / (sumsq[0].sqrt() + 1e-6), max=1.0)
    assert torch.equal(norm, sumsq[0].sqrt())
    # one fp32 division and one product per value: a few ulp
    torch.testing.assert_close(g, want * factor, rtol=1e-6, atol=0)
    assert scale > 0.5 or torch.equal(g, want)


def test_grad_clip_spreads_nan():
    g = torch.ones(1000, device='cuda')
    ulm_ops.grad_clip_(g, torch.tensor([float('nan'), 0.0], device='cuda'), 1.0)
    assert bool(g.isnan().all())
