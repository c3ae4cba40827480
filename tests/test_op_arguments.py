"""Which arguments the ops take and which they refuse; refusals are decided on the host, before any launch."""
import numpy as np
import pytest
import torch

import flash_attn_v100_cuda as fa
import ulm_infer
import ulm_model


@pytest.mark.parametrize('half', ['cos', 'sin'])
def test_causal_attention_wants_both_tables_or_none(half):
    with pytest.raises(ValueError, match='given together'):
        ulm_infer.causal_attention(torch.zeros(1, 4, 192, dtype=torch.float16), 1, **{half: torch.zeros(4, 64)})


@pytest.mark.gpu
@pytest.mark.parametrize('L', [67, 300])
@pytest.mark.parametrize('rope', [True, False])
@pytest.mark.parametrize('form', ['columns of a wider tensor', 'every other row', 'one sequence of a batch'])
def test_causal_attention_reads_strided_projections_in_place(form, L, rope):
    H, w = 2, 3 * 2 * 64
    g = torch.Generator(device='cuda').manual_seed(L)
    cos, sin = (torch.randn(L, 128, generator=g, device='cuda') for _ in range(2)) if rope else (None, None)
    if form == 'columns of a wider tensor':
        qkv = torch.randn(3, L, w + 64, generator=g, device='cuda').half()[..., :w]
    elif form == 'every other row':
        qkv = torch.randn(3, 2 * L, w, generator=g, device='cuda').half()[:, ::2]
    else:
        qkv = torch.randn(L, 3, w, generator=g, device='cuda').half().transpose(0, 1)[1:2]
    for a, b in zip(ulm_infer.causal_attention(qkv, H, cos, sin), ulm_infer.causal_attention(qkv.contiguous(), H, cos, sin)):
        assert torch.equal(a, b)


@pytest.mark.parametrize('qkv,kw', [
    (torch.zeros(0, 5, 7, dtype=torch.float16), {}),                             # an empty tensor of another width
    (torch.zeros(0, 5, 192), {}),                                                # of a type the op does not take
    (torch.zeros(8, 192, dtype=torch.float16), dict(flat_shape=(0, -3))),        # negative sizes
    (torch.zeros(8, 7, dtype=torch.float16), dict(flat_shape=(0, 4))),
    (torch.zeros(0, 5, 192, dtype=torch.float16), dict(cos2d=torch.zeros(5, 64))),
])
def test_qkv_attention_checks_empty_inputs_like_others(qkv, kw):
    with pytest.raises(ValueError):
        fa.qkv_rope_flash_attn(qkv, 1, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize('shape,kw', [((0, 5, 384), {}), ((3, 0, 384), {}), ((8, 384), dict(flat_shape=(0, 4)))])
def test_qkv_attention_of_nothing_is_zero_and_differentiable(shape, kw):
    qkv = torch.ones(shape, dtype=torch.float16, device='cuda', requires_grad=True)
    out = fa.qkv_rope_flash_attn(qkv, 2, **kw)
    assert out.shape == (*shape[:-1], 128) and not out.any()
    assert not torch.autograd.grad(out.sum(), qkv)[0].any()


def test_what_stands_in_for_a_dropout_is_called():
    x, seen = torch.ones(3), []
    hooked = torch.nn.Dropout(0.0)
    hooked.register_forward_hook(lambda m, a, y: seen.append(1))

    class Mine(torch.nn.Dropout):
        def forward(self, t):
            return t + 1

    assert ulm_model._drop(torch.nn.Identity(), x) is x
    assert torch.equal(ulm_model._drop(hooked, x), x) and seen == [1]
    assert torch.equal(ulm_model._drop(Mine(0.0), x), x + 1)
    assert ulm_model._drop(torch.nn.Dropout(0.0), x) is x and ulm_model._drop(torch.nn.Dropout(0.5).eval(), x) is x
    assert not torch.equal(ulm_model._drop(torch.nn.Dropout(1.0), x), x)


@pytest.mark.parametrize('window', [[3, 4, 5], (3, 4, 5), [3.0, 4.0, 5.0], torch.tensor([3, 4, 5]), torch.tensor([3, 4, 5], dtype=torch.int32),
                                    np.array([3, 4, 5], dtype=np.int32), np.array([3.0, 4.0, 5.0]), [torch.tensor(3), torch.tensor(4), torch.tensor(5)], range(3, 6)])
def test_windows_of_any_sequence_type(window):
    ids = ulm_infer._ids(window)
    assert ids.dtype == np.int64 and ids.tolist() == [3, 4, 5]


class _Embeds(torch.nn.Module):
    def __init__(self, V, d):
        super().__init__()
        g = torch.Generator().manual_seed(V)
        self.embedding, self.fc_out = torch.nn.Embedding(V, d), torch.nn.Linear(d, V, bias=False)
        for p in self.parameters():
            p.data = torch.randn(p.shape, generator=g)

    def forward_hidden(self, ids):
        return self.embedding(ids)


@pytest.mark.gpu
@pytest.mark.parametrize('V,d', [(100, 64), (96, 40)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float16])
@pytest.mark.parametrize('kind', ['lists', 'device tensors'])
def test_scores_of_a_module_of_any_width_and_type(V, d, dtype, kind):
    m = _Embeds(V, d).cuda()
    g = torch.Generator().manual_seed(1)
    windows = [torch.randint(0, V, (n,), generator=g).tolist() for n in (1, 2, 9, 30)]
    windows[2][-1] = -100                                 # an ignored label: no loss and no token
    got = ulm_infer.score_windows(m, windows if kind == 'lists' else [torch.tensor(w).cuda() for w in windows], 0, torch.device('cuda'), 3, 7, amp_dtype=dtype)
    for i, w in enumerate(windows):
        x, y = torch.tensor(w[:-1], dtype=torch.long), torch.tensor(w[1:], dtype=torch.long)
        z = (m.embedding.weight.cpu()[x].to(dtype).float() @ m.fc_out.weight.detach().cpu().to(dtype).float().t()).to(dtype).float()
        want = torch.nn.functional.cross_entropy(z, y, ignore_index=-100, reduction='sum') if len(y) else torch.zeros(())
        assert got[1][i] == int((y != -100).sum())
        # logits up to 30 with one rounding to fp16 each
        assert abs(got[0][i] - float(want)) <= 2.0 ** -6 * max(1, len(y))
        assert abs(got[2][i] - int((z.argmax(1) == y).sum())) <= (1 if dtype == torch.float16 else 0)
