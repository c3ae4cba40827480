"""What the native ops owe autograd: checkpointing, saved-tensor hooks and the other uses a differentiable op has."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

import ulm_ops


def _weights(dtype=torch.float32, device='cpu', n=2, d=16):
    g = torch.Generator().manual_seed(3)
    return [torch.nn.Parameter((torch.randn(d, d, generator=g) * d ** -0.5).to(dtype).to(device)) for _ in range(n)]


BLOCKS = {
    'relu': lambda x, w: ulm_ops.linear(ulm_ops.linear(x, w[0]).relu(), w[1]),
    'silu gate': lambda x, w: ulm_ops.linear(torch.nn.functional.silu(ulm_ops.linear(x, w[0])) * x, w[1]),
    'dropout': lambda x, w: ulm_ops.linear(torch.nn.functional.dropout(ulm_ops.linear(x, w[0]), 0.5), w[1]),
    'view': lambda x, w: ulm_ops.linear(ulm_ops.linear(x, w[0]).view(2, -1, 16), w[1]),
}


@pytest.mark.parametrize('frozen', [False, True])
@pytest.mark.parametrize('block', list(BLOCKS))
def test_checkpoint_recomputes_the_same_graph(block, frozen):
    w = _weights()
    w[1].requires_grad_(not frozen)
    x = torch.randn(6, 16, generator=torch.Generator().manual_seed(4))
    wrt = [p for p in w if p.requires_grad]

    def run(call):
        torch.manual_seed(7)
        t = x.clone().requires_grad_()
        return torch.autograd.grad(call(t).square().sum(), [t, *wrt])

    plain = run(lambda t: BLOCKS[block](t, w))
    for a, b in zip(run(lambda t: checkpoint(BLOCKS[block], t, w, use_reentrant=False)), plain):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_checkpoint_with_library_ops_between():
    w = _weights(device='cuda')
    n1 = torch.nn.Parameter(torch.ones(16, device='cuda'))

    def block(x):
        h = ulm_ops.rms_norm(x, n1)
        return x + ulm_ops.linear(torch.tanh(ulm_ops.gated_linear(h, w[0], w[1])), w[0])

    x = torch.randn(32, 16, device='cuda')

    def run(call):
        t = x.clone().requires_grad_()
        with torch.autocast('cuda', dtype=torch.bfloat16):
            y = call(t)
        return torch.autograd.grad(y.float().square().sum(), [t, n1, *w])

    plain = run(block)
    for a, b in zip(run(lambda t: checkpoint(block, t, use_reentrant=False)), plain):
        assert torch.equal(a, b)


@pytest.mark.parametrize('shape', [(3, 4), (2, 3, 4)])
def test_linear_has_second_derivatives(shape):
    g = torch.Generator().manual_seed(5)
    x, w = (torch.randn(s, generator=g, dtype=torch.double, requires_grad=True) for s in (shape, (5, 4)))
    assert torch.autograd.gradgradcheck(ulm_ops.linear, (x, w))


def _tangent(x, w):
    import torch.autograd.forward_ad as fwd
    with fwd.dual_level():
        return ulm_ops.linear(fwd.make_dual(x, torch.ones_like(x)), w)


@pytest.mark.parametrize('transform', [
    _tangent,
    lambda x, w: torch.func.vmap(lambda t: ulm_ops.linear(t, w))(x),
    lambda x, w: torch.func.grad(lambda t: ulm_ops.linear(t, w).sum())(x),
    lambda x, w: torch.func.jvp(lambda t: ulm_ops.linear(t, w), (x,), (x,)),
])
def test_transforms_without_a_rule_are_refused(transform):
    with pytest.raises((RuntimeError, NotImplementedError), match='autograd.Function'):
        transform(torch.ones(3, 2, 16), _weights()[0])


class _Traced(torch.nn.Module):
    def __init__(self, device):
        super().__init__()
        self.w1, self.w3 = _weights(device=device)
        self.scale = torch.nn.Parameter(torch.ones(16, device=device))
        self.device = device

    def forward(self, x):
        if self.device == 'cpu':
            return ulm_ops.linear(x, self.w1).relu()
        h = ulm_ops.rms_norm(x, self.scale)
        x, h = ulm_ops.add_rms_norm(x, ulm_ops.gated_linear(h, self.w1, self.w3).half(), self.scale)
        return x + ulm_ops.swiglu(ulm_ops.linear(h.float(), self.w1), h.float())


@pytest.mark.parametrize('device', ['cpu', pytest.param('cuda', marks=pytest.mark.gpu)])
def test_traced_ops_run_again_on_other_inputs(device):
    m = _Traced(device)
    traced = torch.jit.trace(m, torch.randn(8, 16, device=device))
    x = torch.randn(24, 16, device=device)
    got, want = traced(x), m(x)
    assert torch.equal(got, want)
    a, b = torch.autograd.grad(got.sum(), m.w1)[0], torch.autograd.grad(want.sum(), m.w1)[0]
    # the trace's own backward of the cast to fp16 rounds at another place: one fp16 rounding of a summand
    assert float((a - b).norm()) <= 2.0 ** -11 * float(b.norm())


class _Cut(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


def test_an_input_no_gradient_reaches_has_a_zero_one():
    x, w = torch.randn(3, 16, requires_grad=True), _weights()[0]
    _Cut.apply(ulm_ops.linear(x, w)).sum().backward()
    assert torch.equal(x.grad, torch.zeros(3, 16)) and torch.equal(w.grad, torch.zeros(16, 16))


@pytest.mark.gpu
def test_the_norm_weight_of_an_unused_norm_has_a_zero_gradient():
    x, w = torch.randn(3, 64, device='cuda', requires_grad=True), torch.ones(64, device='cuda', requires_grad=True)
    b = torch.randn(3, 64, device='cuda', dtype=torch.float16, requires_grad=True)
    x_new, _ = ulm_ops.add_rms_norm(x, b, w)
    dx, db, dw = torch.autograd.grad(x_new.sum(), [x, b, w])
    assert torch.equal(dx, torch.ones_like(x)) and torch.equal(db, torch.ones_like(b)) and not dw.any() and dw.shape == w.shape
