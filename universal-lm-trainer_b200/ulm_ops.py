"""RMSNorm, the SwiGLU gate and chunked cross-entropy on the sm_100a library, as autograd ops.

The reference has no custom kernels for these: ``FusedRMSNorm`` calls
F.rms_norm (train.py:1862-1875) and ``compute_loss`` loops fc_out +
F.cross_entropy over row chunks (train.py:2059-2082).  The classes and functions
below keep those names and argument meanings.
"""
import contextlib
import ctypes as C

import torch
import torch.nn as nn

import _native as N

_DT = {torch.float16: N.ULM_F16, torch.bfloat16: N.ULM_BF16, torch.float32: N.ULM_F32}
_16BIT = (torch.float16, torch.bfloat16)


def _stream(t=None):
    """torch's current stream on the tensor's device (or the current device)."""
    return N.current_stream(t.device.index if t is not None and t.device.index is not None else torch.cuda.current_device())


def rms_norm(x, weight, eps: float = 1e-6, out_dtype=None):
    """``weight * x * rsqrt(mean(x^2, -1) + eps)``; fp32 reduction.  The output has x's dtype,
    except that an fp32 x under CUDA autocast gives the autocast dtype directly: F.rms_norm
    (train.py:1872) would return fp32 there and the Linear that follows would round it to 16 bits,
    so rounding the fp32 result once in the kernel yields the same values and saves the cast pass
    (and, in the backward, the cast of the 16-bit gradient back to fp32).  ``out_dtype`` overrides."""
    return N.ext().rms_norm(x, weight, eps, out_dtype)


def add_rms_norm(x, branch, weight, eps: float = 1e-6):
    """The residual add in front of a norm fused with that norm: ``x_new = x + branch`` (train.py:1989,
    1993) and ``y = rms_norm(x_new)`` (the next norm: train.py:1991, 1988 of the following block, or 2054)
    in one pass over memory; returns ``(x_new, y)``.  x is the fp32 residual stream, branch the 16-bit
    output of the attention or feed-forward projection under autocast; x_new is fp32 and y has branch's
    dtype -- the values the unfused sequence (add in fp32, F.rms_norm in fp32, autocast's cast in front
    of the next Linear) produces.  The backward adds the gradient arriving at x_new to rms_norm's and
    writes the sum once, as the fp32 gradient of x and, rounded, as the 16-bit gradient of branch."""
    return N.ext().add_rms_norm(x, branch, weight, eps)


class FusedRMSNorm(nn.Module):
    """train.py:1862-1875."""

    def __init__(self, d_model: int, eps: float = 1e-6):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(d_model))
        self.eps = eps

    def forward(self, x):
        return rms_norm(x, self.weight, self.eps)

    def add_forward(self, x, branch):
        """(x + branch, norm(x + branch)); the fused kernel when the tensors have the training layout
        (fp32 residual stream, 16-bit branch, d <= 1024), the two separate ops otherwise."""
        if (x.is_cuda and x.dtype == torch.float32 and branch.dtype in _16BIT and x.shape[-1] <= 1024
                and x.shape[-1] % 4 == 0 and torch.is_autocast_enabled('cuda')
                and torch.get_autocast_dtype('cuda') == branch.dtype):
            return add_rms_norm(x, branch, self.weight, self.eps)
        x = x + branch
        return x, rms_norm(x, self.weight, self.eps)


def swiglu(a, b):
    """``F.silu(a) * b`` (the gate of train.py:1966-1975's feed-forward) in one kernel each way."""
    return N.ext().swiglu(a, b)


# ---------------------------------------------------------------------------
# Bias-free linear layers with the weight gradient accumulated where it lives
# ---------------------------------------------------------------------------
@contextlib.contextmanager
def wgrad_in_place(enabled=True):
    """While active, `linear` and `chunked_cross_entropy` add their weight gradients straight into an
    existing fp32 ``weight.grad`` with one GEMM (16-bit operands, fp32 accumulation and output, beta = 1)
    instead of returning a 16-bit product that autograd casts and adds in two more passes per parameter
    and micro-batch.  The caller owns the gradient buffers (they must exist, be zeroed per step, and no
    post-accumulate hook may be waiting for these parameters): `ulm_dp.DataParallelStep` does.  It holds for the
    calling thread and the backward passes it starts inside."""
    token = N.ext().enter_wgrad_in_place(bool(enabled)) if N.have_ext() else None
    try:
        yield
    finally:
        if token is not None:
            token.leave()


@contextlib.contextmanager
def weight_cast_scope(copies=None):
    """While active in the calling thread, `linear` keeps the 16-bit copy it makes of a weight and reuses it: the caller promises
    that the weights do not change inside the scope (one optimiser step's forward/backward calls).  Nothing
    is reused across scopes or outside one -- a parameter's version counter cannot be relied on for that
    (fused optimisers update parameters without bumping it).  ``copies``: a `weight_copies` object, which is
    refreshed here; without it each weight is cast on first use."""
    if copies is not None:
        copies.refresh()
    token = N.ext().enter_casts(copies) if N.have_ext() else None
    try:
        yield
    finally:
        if token is not None:
            token.leave()


def weight_copies(weights, dtype):
    """One buffer for the 16-bit copies of ``weights`` (fp32 CUDA parameters), kept by the caller and filled by one fused
    cast each time a `weight_cast_scope` opens with it; weights that follow one another in the list do so in the
    buffer, so that `gated_linear` runs its two projections as one GEMM.  Holds 2 bytes per weight element."""
    return N.ext().WeightCopies(list(weights), dtype)


def linear_copies(model, dtype):
    """`weight_copies` of the fp32 CUDA weights of ``model``'s linear layers (each once); None if there are none."""
    ws = {id(m.weight): m.weight for m in model.modules() if isinstance(m, nn.Linear)}
    ws = [w for w in ws.values() if w.is_cuda and w.dtype == torch.float32]
    return weight_copies(ws, dtype) if ws and dtype in _16BIT else None


def gated_linear(x, w1, w3):
    """``swiglu(linear(x, w1), linear(x, w3))`` (train.py:1975) as one op: both projections write the halves of one
    [rows, 2 d_ff] matrix, which the gate's kernels read and differentiate in place of two."""
    return N.ext().gated_linear(x, w1, w3)


def linear(x, weight):
    """``x @ weight.T`` for the model's bias-free projections (train.py:1925-1926, 1969-1971) in the autocast
    dtype; see `wgrad_in_place` for what it does differently from ``nn.Linear`` in the backward.  On the CPU it needs no
    build of the library."""
    if not x.is_cuda and not N.have_ext():
        return nn.functional.linear(x, weight.to(x.dtype))
    return N.ext().linear(x, weight)


def ce_rows_forward(logits, target, ignore_index):
    """One logits tile [rows, V] -> (lse[rows], loss[rows]) in fp32."""
    lib = N.lib()
    rows, V = logits.shape
    lse = torch.empty((rows,), dtype=torch.float32, device=logits.device)
    loss = torch.empty((rows,), dtype=torch.float32, device=logits.device)
    a = N.CeFwdArgs(logits.data_ptr(), target.data_ptr(), lse.data_ptr(), loss.data_ptr(),
                    logits.stride(0), rows, V, _DT[logits.dtype], int(ignore_index), _stream())
    N.check(lib.ulm_ce_fwd(C.byref(a)), 'cross-entropy forward')
    return lse, loss


def lm_head_lse(hidden, weight, target=None, ignore_index=0, keep_logits=True):
    """The lm-head GEMM with the loss statistics taken in its epilogue (one tcgen05 kernel + a per-row
    finishing kernel): hidden [rows, d] and weight [V, d], both fp16 or both bf16 ->
    (lse [rows] fp32, loss [rows] fp32 or None, logits [rows, V] in the operands' dtype or None).
    With ``keep_logits`` the rounded logits are stored (the backward turns them into their gradient) and the
    per-row loss lse - z[target] is returned; without, only lse."""
    return N.ext().lm_head_lse(hidden, weight, target, int(ignore_index), bool(keep_logits))


def lm_head_score(hidden, weight, target, ignore_index=-100):
    """`lm_head_lse` for scoring: the per-row loss lse - z[target] (fp32, 0 on ignored rows) and whether the target has
    the row's largest logit (uint8; the lowest column counts on ties, as in ``argmax``).  The logits are never stored:
    the epilogue picks the target's and the largest out of the accumulator."""
    return N.ext().lm_head_score(hidden, weight, target, int(ignore_index))


def ce_rows_backward_(logits, target, lse, gscale_dev, ignore_index, gscale=1.0):
    """In place: logits <- (softmax - onehot) * gscale * gscale_dev[0] (0 on ignored rows)."""
    lib = N.lib()
    rows, V = logits.shape
    a = N.CeBwdArgs(logits.data_ptr(), target.data_ptr(), lse.data_ptr(),
                    gscale_dev.data_ptr() if gscale_dev is not None else None, float(gscale),
                    logits.stride(0), rows, V, _DT[logits.dtype], int(ignore_index), _stream())
    N.check(lib.ulm_ce_bwd(C.byref(a)), 'cross-entropy backward')
    return logits


# Largest [rows, V] 16-bit logits buffer the cross-entropy keeps between forward and backward.  Up to this size
# (2.1 GB for the 32768-row token budget at V = 32000: small change on a 180 GB part) the backward turns the
# kept logits into their gradient in place and runs ONE GEMM each for dH and dW over all rows; beyond it the
# loss falls back to the reference's chunk-by-chunk form, recomputing each chunk's logits in the backward.
KEEP_LOGITS_BYTES = 8 << 30

# The kept form takes its logits and their log-sum-exp from ONE kernel (`lm_head_lse`: tcgen05 GEMM with the
# statistics in its epilogue) where the shapes allow (d and V multiples of 64), instead of a library GEMM
# followed by a pass over the logits.  Measured at 32768 x 32000 x 768 in bf16 on B200: 1.44 ms against
# 1.25 + 0.45 ms, identical logits bits.
FUSED_LM_HEAD = True


class _ChunkedCE(torch.autograd.Function):
    """The chunk-by-chunk form of the loss below, for logits beyond KEEP_LOGITS_BYTES: one [chunk_rows, V] tile at a
    time; the forward keeps one fp32 lse per row and the backward recomputes each tile with the lm-head GEMM."""

    @staticmethod
    def forward(ctx, hidden, weight, target, ignore_index, chunk_rows, compute_dtype, denominator):
        rows = hidden.shape[0]
        wc = N.ext().cast_cached(weight, compute_dtype)
        if denominator is None:
            n_tokens = (target != ignore_index).sum().clamp(min=1).float()
        elif torch.is_tensor(denominator):
            n_tokens = denominator.to(device=hidden.device, dtype=torch.float32)
        else:
            # a host number stays a host number: turning it into a device tensor is a pageable host-to-device
            # copy, which makes the launching thread wait for the GPU (measured: 4.6 ms per micro-batch)
            n_tokens = float(denominator)
        lse_all = torch.empty((rows,), dtype=torch.float32, device=hidden.device)
        total = torch.zeros((), dtype=torch.float32, device=hidden.device)
        for i in range(0, rows, chunk_rows):
            tile = hidden[i:i + chunk_rows].to(compute_dtype) @ wc.t()
            lse, loss = ce_rows_forward(tile, target[i:i + chunk_rows], ignore_index)
            lse_all[i:i + chunk_rows] = lse
            total = total + loss.sum()
        ctx.save_for_backward(hidden, weight, target, lse_all, *([n_tokens] if torch.is_tensor(n_tokens) else []))
        ctx.n_tokens = None if torch.is_tensor(n_tokens) else n_tokens
        ctx.ignore_index, ctx.chunk_rows, ctx.compute_dtype = ignore_index, chunk_rows, compute_dtype
        return total / n_tokens

    @staticmethod
    def backward(ctx, gout):
        hidden, weight, target, lse_all, *rest = ctx.saved_tensors
        n_tokens = ctx.n_tokens if ctx.n_tokens is not None else rest[0]
        cd = ctx.compute_dtype
        wc = N.ext().cast_cached(weight, cd)
        g = (gout.float() / n_tokens).reshape(1)
        dh = torch.empty_like(hidden)
        dw = None
        for i in range(0, hidden.shape[0], ctx.chunk_rows):
            hc = hidden[i:i + ctx.chunk_rows].to(cd)
            dl = ce_rows_backward_(hc @ wc.t(), target[i:i + ctx.chunk_rows],
                                   lse_all[i:i + ctx.chunk_rows], g, ctx.ignore_index)
            dh[i:i + ctx.chunk_rows] = dl @ wc
            part = N.ext().weight_grad(weight, dl, hc)     # None: already added into weight.grad
            if part is not None:
                dw = part.float() if dw is None else dw.add_(part)
        return dh, (None if dw is None else dw.to(weight.dtype)), None, None, None, None, None


def chunked_cross_entropy(hidden, weight, target, ignore_index=0, chunk_rows=2048,
                          compute_dtype=None, denominator=None):
    """hidden [rows, d], weight [V, d] (the tied lm head), target int64 [rows]
    -> CE summed over targets != ignore_index and divided by their count
    (train.py:2069-2082), or by ``denominator`` (a number or a tensor) when one is given.

    The reference loops fc_out + F.cross_entropy over row chunks so that no fp32 [rows, V] tensor is ever alive
    (autograd still keeps each chunk's fp32 log-softmax).  Here only 16-bit logits ever exist.  Two forms, same values:
      kept     logits of all rows are produced by one lm-head GEMM into one 16-bit buffer and kept; the
               backward rewrites them in place as (softmax - onehot) * g and runs one GEMM for dH and one
               for dW (no recomputation);
      chunked  one tile of rows at a time with recomputation (`_ChunkedCE`; buffers beyond KEEP_LOGITS_BYTES)."""
    if compute_dtype is None:
        compute_dtype = torch.get_autocast_dtype('cuda') if torch.is_autocast_enabled() else (
            hidden.dtype if hidden.dtype in (torch.float16, torch.bfloat16) else torch.bfloat16)
    if hidden.shape[0] == 0:
        return torch.zeros((), device=hidden.device, requires_grad=True)
    target = target.contiguous()
    if hidden.shape[0] * weight.shape[0] * 2 <= KEEP_LOGITS_BYTES:
        dev = denominator.detach() if torch.is_tensor(denominator) else None
        host, shaped = 0.0, dev is not None and dev.dim() > 0
        if dev is None and denominator is not None:
            host = float(denominator)
            if not host > 0.0:                            # the kernel counts then; a division by this number was asked for
                dev = torch.full((), host, dtype=torch.float32, device=hidden.device)
        elif shaped:                                      # one sum, divided as the tensor's shape says
            dev, host = None, 1.0
        loss = N.ext().kept_cross_entropy(hidden, weight, target, int(ignore_index), compute_dtype, dev, host, FUSED_LM_HEAD)
        return loss / denominator.detach().to(device=hidden.device, dtype=torch.float32) if shaped else loss
    N.ext().check_target(hidden, target)
    return _ChunkedCE.apply(hidden, weight, target, int(ignore_index), int(chunk_rows), compute_dtype, denominator)


def token_targets(ids, labels, padded, ignore_index):
    """The [n, L] ``ids`` as ``padded`` flat rows (0 past the end) and the label each row predicts: the next token of
    its sequence, ``ignore_index`` at a sequence's last position and on the padding rows."""
    out = N.ext().token_targets(ids, labels, padded, int(ignore_index))
    if out is not None:
        return out
    # other integer types, other devices, labels that broadcast: plain torch, whose errors come before any launch
    if labels.is_floating_point():
        raise ValueError('token_targets takes integer labels')
    n, L = ids.shape
    flat = ids.reshape(-1)
    if padded > n * L:
        flat = torch.cat([flat, flat.new_zeros(padded - n * L)])
    target = labels.new_full((padded,), ignore_index, dtype=torch.long)
    target[:n * L].view(n, L)[:, :-1] = labels[:, 1:]
    return flat, target


def grad_clip_(flat_grad, sumsq, max_norm):
    """clip_grad_norm_ on the flat gradients, given their squared norm on the device: scales them by
    min(1, max_norm / (norm + 1e-6)) and returns the norm; no pass over memory when nothing is to be clipped."""
    return N.ext().grad_clip(flat_grad, sumsq, float(max_norm))


_SUMSQ_SCRATCH = {}     # device index -> fp32 scratch for the per-CTA partial sums


def grad_unscale_sumsq_(flat_grad, inv_scale, out2):
    """flat fp32 grads *= inv_scale[0]; out2[0] += sum(g^2); out2[1] = 1 on inf/nan.
    The sum is formed in a fixed order (per-CTA partials, then one CTA), so it is
    bit-identical from call to call on the same values."""
    lib = N.lib()
    scratch = _SUMSQ_SCRATCH.get(flat_grad.device.index)
    if scratch is None:
        scratch = _SUMSQ_SCRATCH[flat_grad.device.index] = torch.empty(
            int(lib.ulm_grad_sumsq_partial_count()), dtype=torch.float32, device=flat_grad.device)
    N.check(lib.ulm_grad_unscale_sumsq(flat_grad.data_ptr(), flat_grad.numel(),
                                       inv_scale.data_ptr() if inv_scale is not None else None,
                                       out2.data_ptr(), scratch.data_ptr(), _stream()), 'grad_unscale_sumsq')
    return out2
