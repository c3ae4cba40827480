"""The attention forward that rotates both Q and K (sequences of at most one query tile), at the edges of its tiles."""
import pytest
import torch

import flash_attn_v100_cuda as fa
import ulm_infer
import ulm_model

pytestmark = pytest.mark.gpu


def _tables(S, heads=2):
    cos, sin = ulm_model.rope_tables(heads * 64, max(S, 1))
    return cos.cuda()[:, :64], sin.cuda()[:, :64]


@pytest.mark.parametrize('S', [1, 31, 63, 64, 65, 67, 127, 128, 129])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16])
def test_same_bits_as_rope_then_attention(S, dtype):
    g = torch.Generator(device='cuda').manual_seed(S)
    B, H = 3, 2
    qkv = torch.randn(B, S, 3 * H * 64, generator=g, device='cuda').to(dtype).requires_grad_()
    do = torch.randn(B, S, H * 64, generator=g, device='cuda').to(dtype)
    cos, sin = _tables(S)
    q, k, v = (t.view(B, S, H, 64).transpose(1, 2) for t in qkv.chunk(3, dim=-1))
    qr, kr = fa.rope(q, k, cos, sin)
    want = fa.flash_attn_v100(qr, kr, v, causal=True).transpose(1, 2).reshape(B, S, H * 64)
    got = fa.qkv_rope_flash_attn(qkv, H, cos, sin, causal=True)
    assert torch.equal(got, want)
    assert torch.equal(torch.autograd.grad(got, qkv, do)[0], torch.autograd.grad(want, qkv, do)[0])
    o, k_out, _ = ulm_infer.causal_attention(qkv.detach(), H, cos, sin)
    assert torch.equal(o, want) and torch.equal(k_out, kr)
    fa.check_status()


@pytest.mark.parametrize('n,S', [(1, 130), (5, 4097), (6, 3600)])
def test_prefill_same_bits_on_both_sides_of_its_size_rule(n, S):
    """Q rotated by the stand-alone launch (up to 20 M elements) or inside the kernel (beyond): the same bits."""
    H = 16
    qkv = torch.randn(n, S, 3 * H * 64, generator=torch.Generator(device='cuda').manual_seed(S), device='cuda').half()
    cos, sin = _tables(S, H)
    q, k, v = (t.view(n, S, H, 64).transpose(1, 2) for t in qkv.chunk(3, dim=-1))
    with torch.no_grad():
        qr, kr = fa.rope(q, k, cos, sin)
        want = fa.flash_attn_v100(qr, kr, v, causal=True).transpose(1, 2).reshape(n, S, H * 64)
    o, k_out, _ = ulm_infer.causal_attention(qkv, H, cos, sin)
    assert torch.equal(o, want) and torch.equal(k_out, kr)
    fa.check_status()


@pytest.mark.parametrize('n,H', [(148, 2), (149, 2), (297, 1), (33, 9), (400, 3)])
@pytest.mark.parametrize('S', [16, 67, 128])
def test_same_bits_on_both_sides_of_the_one_wave_rule(n, H, S):
    """Q and K rotated in their tile (up to 296 CTAs) or by a launch of its own (beyond): the same bits."""
    qkv = torch.randn(n, S, 3 * H * 64, generator=torch.Generator(device='cuda').manual_seed(n + S), device='cuda').half().requires_grad_()
    do = torch.randn(n, S, H * 64, device='cuda').half()
    cos, sin = _tables(S, H)
    q, k, v = (t.view(n, S, H, 64).transpose(1, 2) for t in qkv.chunk(3, dim=-1))
    qr, kr = fa.rope(q, k, cos, sin)
    want = fa.flash_attn_v100(qr, kr, v, causal=True).transpose(1, 2).reshape(n, S, H * 64)
    got = fa.qkv_rope_flash_attn(qkv, H, cos, sin, causal=True)
    assert torch.equal(got, want) and torch.equal(torch.autograd.grad(got, qkv, do)[0], torch.autograd.grad(want, qkv, do)[0])
    o, k_out, _ = ulm_infer.causal_attention(qkv.detach(), H, cos, sin)
    assert torch.equal(o, want) and torch.equal(k_out, kr)
    fa.check_status()
