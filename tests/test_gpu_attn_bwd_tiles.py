"""Attention backward at the edges of its tiles and work lists: query and key tiles of 64 and 128 rows, odd and even numbers of
tiles per work item (the dK/dV kernel's two groups take alternate tiles across items), several items per CTA, items of one tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype,bound', [(torch.float16, 2e-3), (torch.bfloat16, 5e-3)])
@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('B,H,S', [(1, 1, 1), (31, 12, 63), (30, 12, 65), (31, 12, 128), (20, 12, 129), (9, 12, 191), (9, 12, 193), (5, 12, 449)])
def test_backward_at_tile_edges(dtype, bound, causal, B, H, S):
    """Against fp64 softmax attention on the same 16-bit inputs.  P and dS are rounded once to 16 bits before their products and every
    gradient once at the end (2^-9 relative in bf16, 2^-12 in fp16, uncorrelated): norm-wise 2-3e-3 in bf16, 3e-4 in fp16."""
    import flash_attn_v100_cuda as fa
    g = torch.Generator(device='cuda').manual_seed(B * 1000 + S)
    q, k, v, do = (torch.randn((B, S, H, 64), generator=g, device='cuda').to(dtype).transpose(1, 2) for _ in range(4))
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    o = fa.flash_attn_v100(*leaves, causal=causal)
    got = torch.autograd.grad(o, leaves, do)
    fa.check_status()
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = ref[0] @ ref[1].transpose(-1, -2) * 0.125
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device='cuda').triu(1), float('-inf'))
    want = torch.autograd.grad(s.softmax(-1) @ ref[2], ref, do.double())
    for name, a, b in zip(('dq', 'dk', 'dv'), got, want):
        if S == 1 and name != 'dv':                      # one key: the probabilities are constant
            assert float(a.abs().max()) < 1e-3, name
        else:
            assert float((a.double() - b).norm() / b.norm()) <= bound, name
    again = torch.autograd.grad(fa.flash_attn_v100(*leaves, causal=causal), leaves, do)
    assert all(torch.equal(x, y) for x, y in zip(got, again))   # one issuer per accumulator: the same bits on every run
