"""Forward-only use of the attention kernels: the reference's inference model, its perplexity
scoring and its Hugging Face attention module all call F.scaled_dot_product_attention directly
(inf.py:119-135, 866-937; hf_template/modeling_universal_lm.py:117-156).  This module gives the
same three places the sm_100a forward kernel:

    causal_attention(qkv, n_heads, cos, sin)   one causal prefill attention on the fused projection
    patch_attention(model)                     rebinds ``forward`` of every attention module of an
                                               inf.py / HF model (attributes wqkv, wo, n_heads, head_dim)
    score_windows(...)                         inf.py:866-937 with the fused forward and the
                                               cross-entropy row kernel

Only the case the kernel covers is taken over -- causal attention over the whole sequence, no
attention mask, no KV cache, head_dim 64, fp16/bf16 on a B200; anything else (single-token decode
steps with a cache, padded-mask batches, CPU tensors) goes to the module's own forward, which is the
caller's code, not a path of this library.
"""
import array
import types

import numpy as np
import torch

import _native as N
import ulm_model
import ulm_ops


def causal_attention(qkv, n_heads, cos=None, sin=None, softmax_scale=None):
    """qkv [n, L, 3*n_heads*64] 16-bit, rows contiguous -> (attention output [n, L, n_heads*64], k, v) with k
    rotated, both as (n, n_heads, L, 64) views.  ``cos``/``sin``: the model's [1, L, >=64] or [L, >=64]
    fp32 RoPE tables (None: no rotation).  No autograd graph is built and nothing is saved."""
    return N.ext().causal_attention(qkv, n_heads, cos, sin, 64 ** -0.5 if softmax_scale is None else float(softmax_scale))


def _eligible(module, x, mask, past, is_causal):
    return (mask is None and past is None and is_causal and x.is_cuda and not torch.is_grad_enabled()
            and getattr(module, 'head_dim', None) == 64)


def _inf_forward(self, x, mask=None, cos=None, sin=None):
    """Replacement for inf.MultiHeadAttention.forward (inf.py:119-135)."""
    if not _eligible(self, x, mask, None, True):
        return self._ulm_original_forward(x, mask=mask, cos=cos, sin=sin)
    qkv = self.wqkv(x)
    if qkv.dtype not in (torch.float16, torch.bfloat16):
        return self._ulm_original_forward(x, mask=mask, cos=cos, sin=sin)
    out, _, _ = causal_attention(qkv.contiguous(), self.n_heads, cos, sin)
    return self.wo(out)


def _hf_forward(self, x, cos, sin, attention_mask=None, past_key_value=None, use_cache=False, is_causal=True):
    """Replacement for UniversalLMAttention.forward (hf_template/modeling_universal_lm.py:117-156):
    the prefill step; returns (output, (k, v) or None) like the original."""
    if not _eligible(self, x, attention_mask, past_key_value, is_causal):
        return self._ulm_original_forward(x, cos, sin, attention_mask=attention_mask, past_key_value=past_key_value,
                                          use_cache=use_cache, is_causal=is_causal)
    qkv = self.wqkv(x)
    if qkv.dtype not in (torch.float16, torch.bfloat16):
        return self._ulm_original_forward(x, cos, sin, attention_mask=attention_mask, past_key_value=past_key_value,
                                          use_cache=use_cache, is_causal=is_causal)
    out, k, v = causal_attention(qkv.contiguous(), self.n_heads, cos, sin)
    return self.wo(out), ((k, v) if use_cache else None)


def patch_attention(model, style='auto'):
    """Rebind ``forward`` of every attention module of ``model`` -- any submodule with ``wqkv``, ``wo``,
    ``n_heads`` and ``head_dim`` -- to the kernel-backed version.  ``style``: 'inf' for the reference's
    inference model (forward(x, mask, cos, sin)), 'hf' for its Hugging Face module (forward(x, cos, sin,
    attention_mask, past_key_value, use_cache, is_causal)), 'auto' picks 'hf' for modules that carry a
    ``layer_idx``.  Returns the number of modules patched; ``unpatch_attention`` undoes it."""
    n = 0
    for m in model.modules():
        if all(hasattr(m, a) for a in ('wqkv', 'wo', 'n_heads', 'head_dim')) and not hasattr(m, '_ulm_original_forward'):
            kind = style if style != 'auto' else ('hf' if hasattr(m, 'layer_idx') else 'inf')
            m._ulm_original_forward = m.forward
            m.forward = types.MethodType(_hf_forward if kind == 'hf' else _inf_forward, m)
            n += 1
    return n


def unpatch_attention(model):
    for m in model.modules():
        if hasattr(m, '_ulm_original_forward'):
            m.forward = m._ulm_original_forward
            del m._ulm_original_forward


def _ids(window):
    """A window's token ids as an int64 array; a list of Python ints through the array module, which is twice as fast as
    numpy's element-by-element conversion."""
    if isinstance(window, (list, tuple)):
        try:
            return np.frombuffer(array.array('q', window), dtype=np.int64)
        except TypeError:                                 # floats and the like: converted as torch does
            pass
    elif isinstance(window, np.ndarray):
        return window.astype(np.int64, copy=False)
    return torch.as_tensor(window, dtype=torch.long).cpu().numpy()


def score_windows(model, windows, pad_id, device, batch_size, chunk_rows, amp_dtype=torch.float16):
    """inf.py:866-937: per-window (loss sum, token count, correct top-1 count), windows sorted by length
    into right-padded batches, ``input = w[:-1]``, ``label = w[1:]``; ``model`` provides
    ``forward_hidden`` and ``fc_out`` (ulm_model.DecoderOnlyTransformer or the reference's model after
    `patch_attention`).  Only the rows that predict something reach the lm head; where its kernel takes the
    shapes (`ulm_ops.lm_head_score`) the logits are never stored, otherwise they exist for ``chunk_rows`` rows
    at a time.

    The weights do not change inside the call, so their 16-bit copies are made once, and the results of all batches
    come back in one copy: the host launches the next batch while the GPU works on the last one.  48 windows of 192
    to 768 tokens on the 100M preset, fp16: 14.1 -> 8.7 ms."""
    n = len(windows)
    losses, rows_of, correct = [0.0] * n, [max(len(w) - 1, 0) for w in windows], [0] * n
    tokens = list(rows_of)                                # rows whose label is the ignored -100 do not count (it can only come last)
    order = sorted(range(n), key=lambda i: len(windows[i]))
    scored, loss_parts, hit_parts = [], [], []
    on_gpu = torch.device(device).type == 'cuda'
    # the package's own model takes its 16-bit weights from one fused cast; others cast through autocast
    copies = ulm_ops.linear_copies(model, amp_dtype) if isinstance(model, ulm_model.DecoderOnlyTransformer) else None
    with torch.no_grad(), ulm_ops.weight_cast_scope(copies), torch.autocast('cuda', dtype=amp_dtype):
        w16 = None
        for start in range(0, n, batch_size):
            idxs = [i for i in order[start:start + batch_size] if rows_of[i] > 0]
            if not idxs:
                continue
            g, t, m = len(idxs), max(rows_of[i] for i in idxs), sum(rows_of[i] for i in idxs)
            # one copy per batch: the padded inputs, the labels of the rows that predict, and those rows' numbers
            host = torch.full((g * t + 2 * m,), pad_id, dtype=torch.long, pin_memory=on_gpu)
            v = host.numpy()
            at = g * t
            for j, i in enumerate(idxs):
                ids, k = _ids(windows[i]), rows_of[i]
                tokens[i] -= int(ids[-1] == -100)
                v[j * t:j * t + k] = ids[:-1]
                v[at:at + k] = ids[1:]
                v[at + m:at + m + k] = np.arange(j * t, j * t + k)
                at += k
            dev = host.to(device, non_blocking=True)
            input_ids, y, rows = dev[:g * t].view(g, t), dev[g * t:g * t + m], dev[g * t + m:]
            hidden = model.forward_hidden(input_ids)
            h = hidden.reshape(g * t, hidden.shape[-1])
            if m < g * t:
                h = h.index_select(0, rows)
            h = h.to(amp_dtype)
            if w16 is None:
                w16 = N.ext().cast_cached(model.fc_out.weight, amp_dtype)
            if (h.dtype in (torch.float16, torch.bfloat16) and h.shape[1] % 64 == 0 and h.is_contiguous() and w16.is_contiguous()
                    and not (h.data_ptr() | w16.data_ptr()) & 15):
                loss, hit = ulm_ops.lm_head_score(h, w16, y)
                loss_parts.append(loss)
                hit_parts.append(hit)
            else:
                for s in range(0, m, chunk_rows):
                    logits = h[s:s + chunk_rows] @ w16.t()
                    loss_parts.append(ulm_ops.ce_rows_forward(logits, y[s:s + chunk_rows], -100)[1])
                    hit_parts.append((logits.argmax(dim=-1) == y[s:s + chunk_rows]).to(torch.uint8))
            scored += idxs
        if scored:
            loss_rows = torch.cat(loss_parts).cpu().numpy().astype(np.float64)
            hit_rows = torch.cat(hit_parts).cpu().numpy()
            at = 0
            for i in scored:
                k = rows_of[i]
                losses[i] = float(loss_rows[at:at + k].sum())
                correct[i] = int(hit_rows[at:at + k].sum())
                at += k
    return losses, tokens, correct
