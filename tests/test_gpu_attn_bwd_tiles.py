"""Attention backward at the edges of its tiles and work lists: query and key tiles of 64 and 128 rows, odd and even numbers of
tiles per work item (the dK/dV kernel's two groups take alternate tiles across items), several items per CTA, items of one tile."""
import pytest
import torch


@pytest.mark.gpu
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


def tile_error(got, want, rows=64):
    """Largest error of a (batch, head)'s tile of `rows` rows, relative to the tile's own norm or the rms over all heads of that tile's
    norm, whichever is larger (the norm of a single row can come out small by chance)."""
    worst = 0.0
    for r in range(0, want.shape[2], rows):
        w = want[:, :, r:r + rows]
        n = w.norm(dim=(2, 3))
        e = (got[:, :, r:r + rows].double() - w).norm(dim=(2, 3))
        worst = max(worst, float((e / n.clamp_min(float(n.square().mean().sqrt()))).max()))
    return worst


def attention_grads(q, k, v, do, causal, lse_of=None):
    """fp64 gradients.  `lse_of`: for every query row, the row whose softmax statistics are taken for it (None: its own)."""
    q, k, v, do = (t.double() for t in (q, k, v, do))
    S = q.shape[2]
    s = q @ k.transpose(-1, -2) * 0.125
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1), float('-inf'))
    lse = torch.logsumexp(s, -1, keepdim=True)
    dp = do @ v.transpose(-1, -2)
    delta = ((s - lse).exp() * dp).sum(-1, keepdim=True)
    if lse_of is not None:
        lse, delta = lse[:, :, lse_of], delta[:, :, lse_of]
    p = (s - lse).exp()
    ds = p * (dp - delta) * 0.125
    return ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do


# Roundings in series on the way to a gradient: P or dS, O (through delta), the gradient itself, each at most one unit roundoff.
TILE_BOUND = {torch.float16: 3 * 2.0 ** -11, torch.bfloat16: 3 * 2.0 ** -8}


def banded_inputs(B, H, S, dtype, device, seed):
    """Queries whose scale, and with it the softmax statistics, changes from each 64-row tile to the next with a period of five."""
    g = torch.Generator(device=device).manual_seed(seed)
    q, k, v, do = (torch.randn((B, S, H, 64), generator=g, device=device) for _ in range(4))
    q = q * torch.tensor([0.25, 1.5, 0.5, 2.0, 1.0], device=device)[torch.arange(S, device=device) // 64 % 5].view(1, S, 1, 1)
    return [t.to(dtype).transpose(1, 2) for t in (q, k, v, do)]


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('B,H,S', [(1, 2, 1000), (31, 12, 449), (10, 16, 129)])
def test_statistics_reach_their_tile(dtype, causal, B, H, S):
    """dK/dV: the log-sum-exp and delta of a query tile come through shared memory beside the tile, in a ring of six slots.  Neighbouring
    tiles and a slot's successive tiles have different statistics here, so that another tile's would change a key tile's dV by more than its
    bound (test_the_check_sees_stale_statistics)."""
    import flash_attn_v100_cuda as fa
    q, k, v, do = banded_inputs(B, H, S, dtype, 'cuda', S)
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    got = torch.autograd.grad(fa.flash_attn_v100(*leaves, causal=causal), leaves, do)
    fa.check_status()
    for name, a, b in zip(('dq', 'dk', 'dv'), got, attention_grads(q, k, v, do, causal)):
        assert tile_error(a, b) <= TILE_BOUND[dtype], name


@pytest.mark.parametrize('stale', [1, 6])
@pytest.mark.parametrize('causal', [True, False])
def test_the_check_sees_stale_statistics(causal, stale):
    """Any one query tile of sixteen with the statistics of the tile one, or a ring's length, before it."""
    q, k, v, do = banded_inputs(1, 1, 1000, torch.float32, 'cpu', 0)
    want = attention_grads(q, k, v, do, causal)
    for tile in range(6, 16):
        lse_of = torch.arange(1000)
        lse_of[64 * tile:64 * tile + 64] -= 64 * stale
        off = attention_grads(q, k, v, do, causal, lse_of)
        assert tile_error(off[2], want[2]) > 2 * max(TILE_BOUND.values()), tile
