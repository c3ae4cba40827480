"""Attention backward at the edges of its tiles and work lists: query and key tiles of 64 and 128 rows, odd and even numbers of
tiles per work item (the dK/dV kernel's two groups take alternate tiles across items), several items per CTA, items of one tile."""
import pytest
import torch


UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}   # unit roundoff
LEAST = {torch.float16: 2.0 ** -14, torch.bfloat16: 2.0 ** -126, torch.float32: 0.0}   # smallest normal number


def attention_grads(q, k, v, do, causal, lse_of=None):
    """fp64 dQ, dK, dV and, for every row of each, the rms size of its rounding error per unit roundoff.  The kernels round P (forward: for
    O; backward: for dV), O, dS and each gradient once, everything else is fp32; a rounding has an rms of at most 1 / sqrt(3) of the
    unit roundoff (of the smallest normal number where a value is smaller: a last key's dS of 1e-5 was off by eleven times what its own size
    gives in fp16), roundings are independent, and what P and O get in the forward pass reaches dS through delta = sum(O dO) = sum(P dP).
    `lse_of`: for every query row, the row whose softmax statistics are taken for it (None: its own)."""
    least = LEAST[q.dtype] ** 2
    q, k, v, do = (t.double() for t in (q, k, v, do))
    S = q.shape[2]
    s = q @ k.transpose(-1, -2) * 0.125
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1), float('-inf'))
    lse = torch.logsumexp(s, -1, keepdim=True)
    dp = do @ v.transpose(-1, -2)
    p = (s - lse).exp()
    delta = (p * dp).sum(-1, keepdim=True)
    if lse_of is not None:
        lse, delta = lse[:, :, lse_of], delta[:, :, lse_of]
        p = (s - lse).exp()
    ds = p * (dp - delta)
    dq, dk, dv = ds @ k * 0.125, ds.transpose(-1, -2) @ q * 0.125, p.transpose(-1, -2) @ do
    sq = lambda t: t.square().sum(-1, keepdim=True)      # noqa: E731
    var_delta = ((p @ v) * do).square().sum(-1, keepdim=True) + (p * dp).square().sum(-1, keepdim=True)
    var_ds, var_p = (torch.where(p > 0, x.square() + least, 0.0) for x in (ds, p))
    var_q = (var_ds @ sq(k) + var_delta * sq(p @ k)) / 64 + sq(dq)
    var_k = (var_ds + p.square() * var_delta).transpose(-1, -2) @ sq(q) / 64 + sq(dk)
    var_v = var_p.transpose(-1, -2) @ sq(do) + sq(dv)
    return (dq, dk, dv), [((x.squeeze(-1) + 64 * least) / 3).sqrt() for x in (var_q, var_k, var_v)]


def row_error(got, want, rms):
    """Largest error of a row of a (batch, head) over its rms size.  Up to 2e5 rows are looked at: six of them, once in 5e8 for a normal
    variable, are the bound."""
    return float(((got.double() - want).norm(dim=3) / rms).max())


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('B,H,S', [(1, 1, 1), (31, 12, 63), (30, 12, 65), (31, 12, 128), (20, 12, 129), (9, 12, 191), (9, 12, 193), (5, 12, 449)])
def test_backward_at_tile_edges(dtype, causal, B, H, S):
    """Against fp64 softmax attention on the same 16-bit inputs, every row of every head on its own."""
    import flash_attn_v100_cuda as fa
    g = torch.Generator(device='cuda').manual_seed(B * 1000 + S)
    q, k, v, do = (torch.randn((B, S, H, 64), generator=g, device='cuda').to(dtype).transpose(1, 2) for _ in range(4))
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    o = fa.flash_attn_v100(*leaves, causal=causal)
    got = torch.autograd.grad(o, leaves, do)
    fa.check_status()
    for name, a, b, rms in zip(('dq', 'dk', 'dv'), got, *attention_grads(q, k, v, do, causal)):
        assert row_error(a, b, rms) <= 6 * UNIT[dtype], name
    again = torch.autograd.grad(fa.flash_attn_v100(*leaves, causal=causal), leaves, do)
    assert all(torch.equal(x, y) for x, y in zip(got, again))   # one issuer per accumulator: the same bits on every run


@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('S', [63, 65, 129, 191, 193, 449])
def test_the_check_sees_lost_rows(causal, S):
    """In one head of twelve: the last row missing, or the last 64-row tile of another head in its place."""
    g = torch.Generator().manual_seed(S)
    for w, rms in zip(*attention_grads(*(torch.randn((1, 12, S, 64), generator=g) for _ in range(4)), causal)):
        lost, swapped = w.clone(), w.clone()
        lost[0, 5, -1] = 0
        swapped[0, 5, (S - 1) // 64 * 64:] = w[0, 4, (S - 1) // 64 * 64:]
        assert min(row_error(lost, w, rms), row_error(swapped, w, rms)) > 12 * max(UNIT.values())


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
    tiles and a slot's successive tiles have different statistics here, so that another tile's would change some key's dV by more than its
    bound (test_the_check_sees_stale_statistics)."""
    import flash_attn_v100_cuda as fa
    q, k, v, do = banded_inputs(B, H, S, dtype, 'cuda', S)
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    got = torch.autograd.grad(fa.flash_attn_v100(*leaves, causal=causal), leaves, do)
    fa.check_status()
    for name, a, b, rms in zip(('dq', 'dk', 'dv'), got, *attention_grads(q, k, v, do, causal)):
        assert row_error(a, b, rms) <= 6 * UNIT[dtype], name


@pytest.mark.parametrize('stale', [1, 6])
@pytest.mark.parametrize('causal', [True, False])
def test_the_check_sees_stale_statistics(causal, stale):
    """Any one query tile of sixteen with the statistics of the tile one, or a ring's length, before it."""
    q, k, v, do = banded_inputs(1, 1, 1000, torch.float32, 'cpu', 0)
    (_, _, want), (_, _, rms) = attention_grads(q, k, v, do, causal)
    for tile in range(6, 16):
        lse_of = torch.arange(1000)
        lse_of[64 * tile:64 * tile + 64] -= 64 * stale
        assert row_error(attention_grads(q, k, v, do, causal, lse_of)[0][2], want, rms) > 12 * max(UNIT.values()), tile
