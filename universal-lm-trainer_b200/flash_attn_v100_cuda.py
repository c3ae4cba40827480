"""Drop-in for the reference's ``flash_attn_v100_cuda`` module on B200.

Same names, arguments and error behaviour as flash_attn_v100_cuda.py of
sunyi9161/Universal-LM-Trainer (the module train.py:82 imports and calls at
train.py:90,94,100,1912,1913,1950), backed by the sm_100a library
``libulm_b200.so``; the autograd functions are native (csrc/torch_ops.cpp):

    is_available()  build_error()  can_use(q,k,v)
    rope_can_use(q,k,cos2d,sin2d)  rope(q,k,cos2d,sin2d)
    flash_attn_v100(q,k,v,dropout_p=0.0,causal=True,softmax_scale=None)

Differences a caller can see: bf16 is accepted beside fp16; the attention
output has shape (B,H,S,64) like the reference's but is laid out (B,S,H,64) in
memory, so train.py:1963's ``transpose(1,2).contiguous()`` is a no-op; dO may be
strided.  There is no SDPA or CPU path in here: if the library cannot be loaded
the Functions raise, and train.py's own ``if`` decides what to do.

One addition: ``rope_flash_attn(q, k, v, cos2d, sin2d, ...)`` does what
``flash_attn_v100(*rope(q, k, cos2d, sin2d), v, ...)`` does (train.py:1913 +
1950) with the rotation of Q inside the attention forward and the adjoint
rotation of dQ and dK inside the backward's epilogues; only K still goes through
the stand-alone RoPE kernel.  Results are bit-identical to the two-call form.
"""
import ctypes as C
import itertools

import torch

import _native as N

_SEED_COUNTER = itertools.count(1)
_STATUS = {}            # device index -> uint32[1] tensor the kernels OR their timeout bits into


_last_seed = 0          # seed of the most recent forward (tests rebuild the dropout mask from it)


def _next_seed():
    # flash_attn_v100_cuda.py:29-33: the mask is a pure function of the seed, so
    # backward only needs the integer back.
    global _last_seed
    _last_seed = (int(torch.cuda.initial_seed()) * 2654435761 + next(_SEED_COUNTER)) & 0xFFFFFFFF
    return _last_seed


def is_available():
    return N.available()


def build_error():
    return N.build_error()


def _stream(t=None):
    """torch's current stream on the tensor's device (or the current device)."""
    return N.current_stream(t.device.index if t is not None and t.device.index is not None else torch.cuda.current_device())


def _status(dev):
    index = dev.index if dev.index is not None else torch.cuda.current_device()
    s = _STATUS.get(index)
    if s is None:
        s = _STATUS[index] = N.ext().status_tensor(index)
    return s


def check_status(device=None):
    """Raise if any kernel on ``device`` gave up on a barrier wait since the last
    call (synchronises; meant for step boundaries and tests)."""
    dev = torch.device('cuda', torch.cuda.current_device()) if device is None else torch.device(device)
    index = dev.index if dev.index is not None else torch.cuda.current_device()
    s = _status(torch.device('cuda', index))
    bits = int(s.item())
    if bits:
        s.zero_()
        raise RuntimeError(f'attention kernel reported a barrier timeout (status bits {bits:#x})')


def _fa_ready(t):
    """flash_attn_v100_cuda.py:97-102, with bf16 admitted: (B,H,S,64), innermost
    contiguous, 32-byte aligned base and strides."""
    return N.ext().fa_ready(t)


def can_use(q, k, v):
    return N.ext().can_use(q, k, v)


def attn_forward(q, k, v, dropout_p, causal, softmax_scale, seed, cos=None, sin=None, want_q_rot=True, o_out=None):
    """The reference's ``fa_fwd`` (flash_attn_v100.cu:337-364): returns (o, lse, q_rot).
    With ``cos``/``sin`` (fp32 [S,64] views) q is taken unrotated and rotated inside the
    kernel; q_rot is the rotated copy the backward needs (None without tables).  ``o_out``: a
    preallocated (B,H,S,64) view to write the output into."""
    return N.ext().attn_forward(q, k, v, float(dropout_p), bool(causal), float(softmax_scale), int(seed), cos, sin, bool(want_q_rot), o_out)


def _seed_for(dropout_p):
    """The seed of the next forward; without dropout nothing reads it, so only the sequence advances."""
    if dropout_p:
        return _next_seed()
    next(_SEED_COUNTER)
    return 0


class _FlashAttnV100Cuda:
    """flash_attn_v100_cuda.py:69-94: the op itself, without the wrapper's defaults."""

    @staticmethod
    def apply(q, k, v, dropout_p, causal, softmax_scale):
        return N.ext().flash_attn(q, k, v, float(dropout_p), bool(causal), float(softmax_scale), _next_seed())


def attn_backward(q, k, v, o, lse, do, dropout_p, causal, softmax_scale, seed, mode=7,
                  delta=None, cos=None, sin=None, out=None):
    """The reference's ``fa_bwd`` (flash_attn_v100_bwd.cu:433-506): returns
    (dq, dk, dv); ``mode`` selects delta / dQ / dK,dV passes like its bitmask.
    With ``cos``/``sin`` q and k are the rotated tensors and dq, dk come back as the
    gradients of the unrotated ones (adjoint rotation in the kernels' epilogues)."""
    return tuple(N.ext().attn_backward(q, k, v, o, lse, do, float(dropout_p), bool(causal), float(softmax_scale), int(seed), int(mode), delta, cos, sin, out))


def _rope_launch(q, k, cos, sin, backward):
    """The stand-alone kernel or its adjoint; q may be None: only k is rotated then (and None comes back in q's place)."""
    return N.ext().rope_launch(q, k, cos, sin, bool(backward))


class _RopeV100Cuda:
    """flash_attn_v100_cuda.py:111-138: fused RoPE, one kernel each way."""

    @staticmethod
    def apply(q, k, cos, sin):
        return N.ext().rope(q, k, cos, sin)


def rope_can_use(q, k, cos, sin):
    """flash_attn_v100_cuda.py:141-147 (plus the 16-byte table alignment the
    vector loads here need)."""
    return N.ext().rope_can_use(q, k, cos, sin)


def rope(q, k, cos2d, sin2d):
    """q,k: (B,H,S,64) 16-bit views of any stride; cos2d/sin2d: fp32 (S,64), rows may be padded."""
    return N.ext().rope(q, k, cos2d, sin2d)


def flash_attn_v100(q, k, v, dropout_p: float = 0.0, causal: bool = True, softmax_scale=None):
    """flash_attn_v100_cuda.py:155-166."""
    if softmax_scale is None:
        softmax_scale = q.shape[-1] ** -0.5
    return N.ext().flash_attn(q, k, v, dropout_p, bool(causal), softmax_scale, _seed_for(dropout_p))


# Where the RoPE work of rope_flash_attn / qkv_rope_flash_attn runs.  All three give the same bits.
#   'none'  stand-alone RoPE kernel on q and k, plain attention kernels, stand-alone RoPE adjoint kernel
#   'fwd'   Q rotated inside the attention forward (K through the stand-alone kernel), backward as 'none'
#   'all'   as 'fwd', and the adjoint applied in the dQ / dK epilogues of the backward kernels
# The kernels of one call on B200, us, none / fwd / all: 8x12x4096 bf16 1158 / 1160-1190 / 1256-1261, 24x12x1363 fp16 586-611 / 584-600 /
# 604-616, 64x12x300 bf16 222-227 / 234 / 263-266, 4x12x201 fp16 30.5 / 31.6 / 32.0.  The forward fusion costs what it saves (the
# rotation sits on each CTA's start-up path).  The backward fusion costs more than the launch it removes, although the dQ epilogue
# runs under the SM's other CTA and the dK epilogue in a warpgroup of its own, whose registers spill.  So 'none' is the default; where
# the host is the limit (4x12x201) 'all', with fewer launches, is 5 % faster a call.
ROPE_FUSION = 'none'
_FUSE = {'none': 0, 'fwd': 1, 'all': 2}


def _fuse_code(fuse):
    code = _FUSE.get(ROPE_FUSION if fuse is None else fuse)
    if code is None:
        raise ValueError("fuse must be 'none', 'fwd' or 'all'")
    return code


def _rope_attn_forward(q, k, v, cos, sin, dropout_p, causal, softmax_scale, seed, fuse):
    """-> (o, lse, q_rot, k_rot): what `rope_flash_attn` launches, without a graph"""
    return tuple(N.ext().rope_attn_forward(q, k, v, cos, sin, float(dropout_p), bool(causal), float(softmax_scale), int(seed), _fuse_code(fuse)))


def _rope_attn_backward(q_rot, k_rot, v, o, lse, do, cos, sin, dropout_p, causal, softmax_scale, seed, fuse):
    """-> (dq, dk, dv) of the UNROTATED q, k and of v"""
    return tuple(N.ext().rope_attn_backward(q_rot, k_rot, v, o, lse, do, cos, sin, float(dropout_p), bool(causal), float(softmax_scale), int(seed), _fuse_code(fuse)))


def rope_flash_attn(q, k, v, cos2d, sin2d, dropout_p: float = 0.0, causal: bool = True, softmax_scale=None, fuse=None):
    """``flash_attn_v100(*rope(q, k, cos2d, sin2d), v, ...)`` as one op (see the module docstring);
    ``fuse`` picks where the RoPE work runs (default: ROPE_FUSION).  Inputs must satisfy
    ``rope_can_use`` and ``can_use``; there is no other path."""
    if softmax_scale is None:
        softmax_scale = q.shape[-1] ** -0.5
    return N.ext().rope_flash_attn(q, k, v, cos2d, sin2d, dropout_p, bool(causal), softmax_scale, _seed_for(dropout_p), _fuse_code(fuse))


def qkv_rope_flash_attn(qkv, n_heads, cos2d=None, sin2d=None, dropout_p: float = 0.0, causal: bool = True,
                        softmax_scale=None, fuse=None, flat_shape=None):
    """qkv [n, L, 3*n_heads*64] (the fused projection, 16-bit, contiguous) -> attention output
    [n, L, n_heads*64]; RoPE with the fp32 (L,64) tables when they are given.  With ``flat_shape=(n, L)``
    qkv is the flattened [T', 3*n_heads*64] tensor with T' >= n*L (padding rows at the end) and the output is
    [T', n_heads*64] with zero padding rows: no copy either way.

    This is the attention block between the two projections of train.py:1934-1964 as one op: chunk into q, k, v
    (train.py:1935-1939), RoPE on q and k, causal attention, heads merged back (train.py:1963).  Nothing is copied
    that the reference copies around the kernels: q, k, v are strided views of qkv, the output comes out of the kernel
    in (n, L, H, 64) order, and the backward kernels write dq, dk, dv straight into the three slices of one gradient
    tensor (autograd would otherwise concatenate them)."""
    n, L = (-1, -1) if flat_shape is None else flat_shape
    if flat_shape is not None and min(n, L) < 0:
        raise ValueError('flat_shape=(n, L) takes sizes')
    code = _fuse_code(fuse)
    if softmax_scale is None:
        softmax_scale = 64 ** -0.5
    return N.ext().qkv_attn(qkv, n_heads, cos2d, sin2d, dropout_p, bool(causal), softmax_scale, _seed_for(dropout_p), code, n, L)


def selftest_wait_timeout(limit_ns=2_000_000, device=None):
    """Launch the library's wait self-test: one bounded barrier wait of ``limit_ns`` on a
    barrier nothing arrives at.  The kernel returns by itself and leaves the timeout bit
    in the device's status word, where ``check_status`` finds it."""
    dev = torch.device('cuda', torch.cuda.current_device()) if device is None else torch.device(device)
    N.check(N.lib().ulm_selftest_wait_timeout(int(limit_ns), _status(dev).data_ptr(), _stream()), 'selftest_wait_timeout')


def tensor_map_cache_stats():
    """(hits, misses) of the library's cache of encoded TMA tensor maps."""
    h, m = C.c_uint64(0), C.c_uint64(0)
    N.lib().ulm_tensor_map_cache_stats(C.byref(h), C.byref(m))
    return int(h.value), int(m.value)
