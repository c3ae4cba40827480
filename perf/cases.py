"""The work whose speed matters to a user of this package, as cases that can be timed and compared.

A case is a dict of plain values.  ``prepare`` makes what a program has in hand before the call, ``run`` makes one
pass through the public entry points, ``work`` says what the pass cannot do without and ``tolerance`` how far another
correct implementation of the same precision may differ.  Kinds:

  attn     RoPE + causal attention, forward and backward, by one of the three calls a training program makes:
           'dropin' (rope, then flash_attn_v100, on views of the fused projection), 'fused' (rope_flash_attn on
           separate tensors) or 'qkv' (qkv_rope_flash_attn, what ulm_model calls per layer)
  prefill  ulm_infer.causal_attention: the forward alone, no graph, as the inference modules call it
  norm     RMSNorm forward and backward; 'add' is the training layout (fp32 residual stream + 16-bit branch)
  gate     the SwiGLU gate, forward and backward
  loss     chunked_cross_entropy (lm head + loss), forward and backward
  step     one optimiser step of DataParallelStep on a preset of ulm_train
  score    ulm_infer.score_windows: perplexity scoring of token windows
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath('universal-lm-trainer_b200')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import flash_attn_v100_cuda as fa  # noqa: E402
import ulm_dp  # noqa: E402
import ulm_infer  # noqa: E402
import ulm_model  # noqa: E402
import ulm_ops  # noqa: E402
import ulm_train  # noqa: E402

_DTYPES = {'fp16': torch.float16, 'bf16': torch.bfloat16}


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the headline attention benchmark: 8 sequences of the longest context
        dict(name='attn_4096', kind='attn', call='fused', n=8, heads=12, length=4096, dtype='bf16'),
        # one layer of a token-budget micro-batch (about 32768 tokens) of the 100M preset, fp16 as it is trained;
        # padded length and row count are whatever the bucket gave
        dict(name='attn_micro_batch', kind='attn', call='qkv', n=24, heads=12, length=1363, dtype='fp16'),
        # the reference trainer's own two calls on a few short sequences: launches and host time count
        dict(name='attn_short', kind='attn', call='dropin', n=4, heads=12, length=201, dtype='fp16'),
        # inference: a long prompt of the scaled preset's width
        dict(name='prefill_4096', kind='prefill', n=1, heads=16, length=4096, dtype='bf16'),
        # inference: a short prompt, where one call's latency is what the user waits for
        dict(name='prefill_short', kind='prefill', n=1, heads=12, length=67, dtype='fp16'),
        # residual add + norm over a full micro-batch, the form every block of a training step runs twice
        dict(name='norm_add', kind='norm', add=True, rows=32768, d=768, dtype='fp16'),
        # a plain norm over a few hundred rows (evaluation batches, inference)
        dict(name='norm_small', kind='norm', add=False, rows=514, d=1024, dtype='bf16'),
        # the feed-forward gate of a full micro-batch
        dict(name='gate', kind='gate', rows=32768, d=2048, dtype='bf16'),
        # lm head + loss of a full micro-batch, 5 % of the targets ignored
        dict(name='loss', kind='loss', rows=32768, d=768, vocab=32000, dtype='bf16'),
        # one optimiser step of the 100M preset over two micro-batches of about 32768 tokens
        dict(name='step_100m', kind='step', preset='100m', micro_batches=2, rows=30, length=1087),
        # one optimiser step of the tiny preset: smoke runs and unit-sized experiments, bound by launches
        dict(name='step_tiny', kind='step', preset='tiny64', micro_batches=1, rows=8, length=256),
        # perplexity scoring of a document set with the 100M preset
        dict(name='score', kind='score', windows=48, length=768, batch=16, chunk_rows=4096, dtype='fp16'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['attn', 'attn', 'attn', 'prefill', 'prefill', 'norm', 'norm', 'gate', 'loss', 'step', 'step', 'score'])
    dtype = rng.choice(['fp16', 'bf16'])
    if kind == 'attn':
        heads, length = rng.choice([2, 12, 16]), _log_int(rng, 32, 4096)
        # from two rows to a full token budget, never more score elements than the headline case
        most = min(64, max(1, 32768 // length), max(1, int(8 * 12 * 4096 ** 2 / (heads * length ** 2))))
        return dict(kind='attn', call=rng.choice(['dropin', 'fused', 'qkv']), n=_log_int(rng, 1, most), heads=heads,
                    length=length, dtype=dtype)
    if kind == 'prefill':
        return dict(kind='prefill', n=rng.choice([1, 1, 2, 4, 8]), heads=rng.choice([2, 12, 16]),
                    length=_log_int(rng, 16, 4096), dtype=dtype)
    if kind == 'norm':
        return dict(kind='norm', add=rng.random() < 0.6, rows=_log_int(rng, 64, 32768), d=rng.choice([128, 768, 1024]), dtype=dtype)
    if kind == 'gate':
        return dict(kind='gate', rows=_log_int(rng, 64, 32768), d=rng.choice([344, 2048, 2816]), dtype=dtype)
    if kind == 'loss':
        d, vocab = rng.choice([(128, 4096), (768, 32000), (768, 32000), (1024, 32000)])
        return dict(kind='loss', rows=_log_int(rng, 256, 24576 if d == 1024 else 32768), d=d, vocab=vocab, dtype=dtype)
    if kind == 'step':
        if rng.random() < 0.5:
            return dict(kind='step', preset='tiny64', micro_batches=rng.choice([1, 2]), rows=_log_int(rng, 2, 64),
                        length=_log_int(rng, 32, 256))
        length = _log_int(rng, 128, 4096)
        return dict(kind='step', preset='100m', micro_batches=rng.choice([1, 2]),
                    rows=_log_int(rng, 1, max(1, min(64, int(26000 / length)))), length=length)
    return dict(kind='score', windows=_log_int(rng, 8, 48), length=_log_int(rng, 64, 768), batch=rng.choice([8, 16]),
                chunk_rows=rng.choice([2048, 4096]), dtype=dtype)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _randn(g, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=g, device='cuda') * std).to(dtype)


def _tables(heads, length):
    cos, sin = ulm_model.rope_tables(heads * 64, length)     # d_model wide; a head reads the first 64 columns
    return cos.cuda()[:, :64], sin.cuda()[:, :64]


def _trainer(case, seed):
    """Model, optimiser and step object as a training program holds them."""
    with torch.device('cuda'):
        model, preset = ulm_train.build(case['preset'], 'cuda', seed=seed)
    # the parameters are slices of one buffer, so that all of the updated state comes back as one tensor
    params = list(model.parameters())
    offsets = np.cumsum([0] + [(p.numel() + 3) // 4 * 4 for p in params])
    flat = torch.zeros(int(offsets[-1]), device='cuda')
    for p, off in zip(params, offsets):
        view = flat[int(off):int(off) + p.numel()].view_as(p)
        view.copy_(p.data)
        p.data = view
    step = ulm_dp.DataParallelStep(model, ulm_train.make_optimizer(model), samples_per_step=case['micro_batches'] * case['rows'],
                                   autocast_dtype=preset['dtype'], loss_scale=preset['loss_scale'])
    return step, flat, preset['model']['vocab_size']


def _micro_batches(case, seed, vocab):
    """Host int64 [n, L] micro-batches as the collate makes them: [BOS] + body + [EOS], bucketed lengths, 0-padded."""
    rng, out = np.random.default_rng(seed), []
    for _ in range(case['micro_batches']):
        n, length = case['rows'], case['length']
        ids = rng.integers(4, vocab, (n, length))
        lens = rng.integers(max(3, int(0.85 * length)), length + 1, n)
        lens[rng.integers(0, n)] = length
        ids[:, 0] = ulm_train.BOS
        ids[np.arange(n), lens - 1] = ulm_train.EOS
        ids[np.arange(length)[None, :] >= lens[:, None]] = ulm_train.PAD
        out.append(torch.from_numpy(ids).pin_memory())
    return out


def prepare(case, seed):
    kind = case['kind']
    g = _gen(seed)
    dtype = _DTYPES.get(case.get('dtype'))
    s = dict(case=case)
    if kind == 'attn':
        n, heads, length = case['n'], case['heads'], case['length']
        s['cos'], s['sin'] = _tables(heads, length)
        if case['call'] == 'fused':
            s['in'] = [_randn(g, (n, heads, length, 64), dtype).requires_grad_() for _ in range(3)]
            s['do'] = _randn(g, (n, heads, length, 64), dtype)
        else:
            s['in'] = [_randn(g, (n, length, 3 * heads * 64), dtype).requires_grad_()]
            s['do'] = _randn(g, (n, length, heads * 64), dtype)
    elif kind == 'prefill':
        s['cos'], s['sin'] = _tables(case['heads'], case['length'])
        s['qkv'] = _randn(g, (case['n'], case['length'], 3 * case['heads'] * 64), dtype)
    elif kind == 'norm':
        rows, d = case['rows'], case['d']
        w = (1.0 + 0.1 * torch.randn(d, generator=g, device='cuda')).requires_grad_()
        x = _randn(g, (rows, d), torch.float32 if case['add'] else dtype).requires_grad_()
        s['in'] = [x, w]
        s['dy'] = _randn(g, (rows, d), dtype)
        if case['add']:
            s['in'].append(_randn(g, (rows, d), dtype).requires_grad_())
            s['dx'] = _randn(g, (rows, d), torch.float32)
    elif kind == 'gate':
        s['in'] = [_randn(g, (case['rows'], case['d']), dtype).requires_grad_() for _ in range(2)]
        s['dy'] = _randn(g, (case['rows'], case['d']), dtype)
    elif kind == 'loss':
        h = _randn(g, (case['rows'], case['d']), dtype).requires_grad_()
        w = _randn(g, (case['vocab'], case['d']), torch.float32, 0.02).requires_grad_()
        t = torch.randint(1, case['vocab'], (case['rows'],), generator=g, device='cuda')
        t[torch.rand(case['rows'], generator=g, device='cuda') < 0.05] = 0
        s['in'], s['target'], s['dtype'] = [h, w], t, dtype
    elif kind == 'step':
        s['step'], s['params'], vocab = _trainer(case, seed)
        s['batches'] = _micro_batches(case, seed, vocab)
    else:
        with torch.device('cuda'):
            s['model'], preset = ulm_train.build('100m', 'cuda', seed=seed)
        s['model'].eval()
        rng = np.random.default_rng(seed)
        lens = rng.integers(max(2, case['length'] // 4), case['length'] + 1, case['windows'])
        lens[0] = case['length']
        s['windows'] = [rng.integers(4, preset['model']['vocab_size'], int(k)).tolist() for k in lens]
        s['dtype'] = dtype
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _run_attn(s):
    case, cos, sin = s['case'], s['cos'], s['sin']
    n, heads, length = case['n'], case['heads'], case['length']
    if case['call'] == 'fused':
        o = fa.rope_flash_attn(*s['in'], cos, sin, causal=True)
    elif case['call'] == 'qkv':
        o = fa.qkv_rope_flash_attn(s['in'][0], heads, cos, sin, causal=True)
    else:
        q, k, v = (t.view(n, length, heads, 64).transpose(1, 2) for t in s['in'][0].chunk(3, dim=-1))
        q, k = fa.rope(q, k, cos, sin)
        o = fa.flash_attn_v100(q, k, v, causal=True).transpose(1, 2).reshape(n, length, heads * 64)
    return [o.detach(), *torch.autograd.grad(o, s['in'], s['do'])]


def run(state):
    s, kind = state, state['case']['kind']
    if kind == 'attn':
        return _run_attn(s)
    if kind == 'prefill':
        o, k, _ = ulm_infer.causal_attention(s['qkv'], s['case']['heads'], s['cos'], s['sin'])
        return [o, k]
    if kind == 'norm':
        if s['case']['add']:
            x, w, branch = s['in']
            x_new, y = ulm_ops.add_rms_norm(x, branch, w, 1e-6)
            return [x_new.detach(), y.detach(), *torch.autograd.grad([x_new, y], s['in'], [s['dx'], s['dy']])]
        y = ulm_ops.rms_norm(*s['in'], 1e-6)
        return [y.detach(), *torch.autograd.grad(y, s['in'], s['dy'])]
    if kind == 'gate':
        y = ulm_ops.swiglu(*s['in'])
        return [y.detach(), *torch.autograd.grad(y, s['in'], s['dy'])]
    if kind == 'loss':
        loss = ulm_ops.chunked_cross_entropy(*s['in'], s['target'], ignore_index=0, chunk_rows=4096, compute_dtype=s['dtype'])
        return [loss.detach(), *torch.autograd.grad(loss, s['in'])]
    if kind == 'step':
        loss, norm, _ = s['step'].step(s['batches'])
        return [loss, norm, s['step'].grads.flat, s['params']]
    case = s['case']
    losses, tokens, correct = ulm_infer.score_windows(s['model'], s['windows'], 0, torch.device('cuda'), case['batch'],
                                                      case['chunk_rows'], amp_dtype=s['dtype'])
    return [np.asarray(losses), np.asarray(tokens), np.asarray(correct)]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case['kind']
    if kind in ('attn', 'prefill'):
        elems = case['n'] * case['heads'] * case['length'] * 64
        scores = case['n'] * case['heads'] * case['length'] ** 2 / 2          # the causal half
        if kind == 'attn':                # q, k, v, dO read; o, dq, dk, dv written; seven products of 2*64 flops per score
            return dict(bytes=8 * 2 * elems, flops=7 * 2 * 64 * scores)
        return dict(bytes=5 * 2 * elems, flops=2 * 2 * 64 * scores)           # q, k, v read; o and the rotated k written
    if kind == 'norm':
        n = case['rows'] * case['d']
        # add: x, g_x fp32 and branch, g_y 16-bit read; x_new, dx fp32 and y, d_branch 16-bit written.  plain: x, dy; y, dx
        return dict(bytes=(24 if case['add'] else 8) * n, flops=0)
    if kind == 'gate':
        return dict(bytes=6 * 2 * case['rows'] * case['d'], flops=0)          # a, b, dy; y, da, db
    if kind == 'loss':                                                        # h, dh; w, dw in fp32; three products
        return dict(bytes=4 * case['rows'] * case['d'] + 8 * case['vocab'] * case['d'],
                    flops=3 * 2 * case['rows'] * case['d'] * case['vocab'])
    preset = '100m' if kind == 'score' else case['preset']
    m = ulm_train.PRESETS[preset]['model']
    params = m['vocab_size'] * m['d_model'] + m['n_layers'] * (4 * m['d_model'] ** 2 + 3 * m['d_model'] * m['d_ff'])
    if kind == 'step':
        tokens = case['micro_batches'] * case['rows'] * case['length']
        # weights, gradients and both moments in fp32: read and written once
        return dict(bytes=32 * params + 8 * tokens, flops=tokens * ulm_train.flops_per_token(preset, case['length']))
    mean = 0.625 * case['length']                                             # lengths are uniform in [1/4, 1]
    tokens = case['windows'] * mean
    return dict(bytes=4 * params + 16 * tokens, flops=tokens * (2 * params + 2 * mean * m['d_model'] * m['n_layers']))


def tolerance(case):
    if case['kind'] == 'step':
        # gradients of a whole network whose activations are 16-bit
        return dict(rel=2e-2 if case['preset'] == 'tiny64' else 1e-2)
    if case['kind'] == 'score':
        # sums of fp32 losses over 16-bit logits; a tie may move a top-1 hit
        return dict(rel=1e-3, differ=0.01)
    return dict(rel=1e-2 if case['dtype'] == 'bf16' else 3e-3)                # one or two 16-bit roundings per output
