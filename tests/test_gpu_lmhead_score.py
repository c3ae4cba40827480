"""The scoring form of the lm-head kernel (ulm_lmhead_score) at the edges of its tiles, work-item split and tie rule."""
import pytest
import torch

import flash_attn_v100_cuda as fa
import ulm_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('rows,V,d', [(1, 1, 64), (1, 257, 64), (127, 64, 128), (129, 4096, 128), (300, 1000, 192), (2048, 4096, 128),
                                      (515, 32000, 768), (20000, 1300, 64)])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
def test_score_matches_the_stored_logits(rows, V, d, dtype):
    g = torch.Generator(device='cuda').manual_seed(rows + V)
    h = torch.randn(rows, d, generator=g, device='cuda').to(dtype)
    w = (torch.randn(V, d, generator=g, device='cuda') * (2.0 * d ** -0.5)).to(dtype)
    w[V // 2] = w[0]                                      # equal logits in two columns: the lower one is the largest
    t = torch.randint(0, V, (rows,), generator=g, device='cuda')
    z = (h.float() @ w.float().t()).to(dtype)
    t[::2] = z.argmax(dim=1)[::2]                         # targets that hit
    t[::7] = -100
    loss, hit = ulm_ops.lm_head_score(h, w, t)
    fa.check_status()
    used = t != -100
    want = torch.where(used, torch.logsumexp(z.float(), 1) - z.float().gather(1, t.clamp(min=0)[:, None])[:, 0], 0.0)
    # one ulp of the largest logit: the kernel's accumulation order may round a logit the other way
    ulp = float(z.float().abs().max()) * 2.0 ** (-7 if dtype == torch.bfloat16 else -10)
    assert float((loss - want).abs().max()) <= ulp + 1e-5
    assert not hit[~used].any()
    # the target is among the largest up to that flip
    zt = z.float().gather(1, t.clamp(min=0)[:, None])[:, 0]
    top = z.float().max(dim=1).values
    assert bool((zt >= top - ulp)[hit.bool()].all())
    assert float((hit.bool() != (used & (z.argmax(dim=1) == t))).float().mean()) <= (0.02 if rows > 100 else 0.0)


def test_score_gives_ties_to_the_lowest_column():
    h = torch.ones(200, 64, device='cuda', dtype=torch.float16)
    w = torch.zeros(900, 64, device='cuda', dtype=torch.float16)
    for c in (130, 131, 500, 899):
        w[c] = 1
    t = torch.tensor([130, 131, 500, 899, 0] * 40, device='cuda')
    _, hit = ulm_ops.lm_head_score(h, w, t)
    assert hit.tolist() == [1, 0, 0, 0, 0] * 40


@pytest.mark.parametrize('V', [1, 64, 300, 4100])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
def test_score_ranks_infinities_and_nans_as_argmax_does(V, dtype):
    inf, nan = float('inf'), float('nan')
    h = torch.zeros(1, 64, dtype=dtype)
    h[0, 0] = 1
    rows = torch.linspace(-1, 1, V).repeat(6, 1)          # finite; all -inf; +inf twice; one NaN; two; nothing but NaN
    rows[1] = -inf
    rows[2, [V // 3, V // 2]] = inf
    rows[3, V - 1] = nan
    rows[4, [V // 2, V - 1]] = nan
    rows[5] = nan
    for row in range(6):
        w = torch.zeros(V, 64, dtype=dtype)
        w[:, 0] = rows[row].to(dtype)
        z = (h.float() @ w.float().t())[0]
        for target in {int(z.argmax()), 0, V // 2, V - 1}:
            _, hit = ulm_ops.lm_head_score(h.cuda(), w.cuda(), torch.tensor([target], device='cuda'))
            assert bool(hit[0]) == (int(z.argmax()) == target), (row, target)
    fa.check_status()
