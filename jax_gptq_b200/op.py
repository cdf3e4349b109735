"""Host-side mirror of the reference's ``jax_gptq/op.py``: the packed-int4 matmul
operator, differentiable with respect to the activations.

``quantized_matmul(x, qm)`` computes ``x @ dequant(qm)`` and, with
``transpose_b=True``, ``x @ dequant(qm)^T`` - the pair the reference wires up as
forward and backward of its ``custom_vjp`` (op.py:19-20, 71-81).  The launch the
reference hands to ``jt.triton_call`` (op.py:46-63) is the single C-ABI call
``jgq_w4_matmul`` here.
"""
from __future__ import annotations

import torch
from torch.autograd import forward_ad

from . import _lib
from ._lib import lib, check
from .gptq import _to_dev, _out, _is_np, _workspace, _DT

_functorch_active = torch._C._functorch.peek_interpreter_stack
_tracing = torch._C._get_tracing_state
_current_device, _raw_stream = torch._C._cuda_getDevice, torch._C._cuda_getCurrentRawStream     # the context exists by then
_ZS = {torch.float32: _lib.F32, torch.float16: _lib.F16}


def _settled(w):
    """True from the second matmul on an unchanged packed-weight tensor: the weights were then complete
    before the kernel enqueued just ahead of this call (at the latest, the previous matmul on them)
    started, which is what JGQ_W4_WEIGHTS_SETTLED promises.  An in-place update through torch bumps the
    tensor's version counter and makes the next call an ordinary one again."""
    seen = getattr(w, '_jgq_seen_version', None)
    w._jgq_seen_version = w._version
    return seen == w._version


_ws_bytes = {}           # (device, M, N, K, transpose_b) -> workspace bytes: a function of the sizes and the device's SM count


def _workspace_bytes(dev, M, N, K, transpose_b):
    """For the current device, whose index is `dev`."""
    key = (dev, M, N, K, transpose_b)
    need = _ws_bytes.get(key)
    if need is None:
        if len(_ws_bytes) >= 4096:
            _ws_bytes.clear()
        need = _ws_bytes[key] = lib.jgq_w4_matmul_workspace_bytes(M, N, K, int(transpose_b))
    return need


def _launch(x, w, zero, scale, transpose_b):
    shape = x.shape
    if len(shape) > 2:                                # op.py:21-24
        x = x.reshape(-1, shape[-1])
    if not x.is_contiguous():
        x = x.contiguous()
    M, K = x.shape
    Kw, Nw = w.shape
    Kw *= 2
    K2, out_n = (Nw, Kw) if transpose_b else (Kw, Nw)    # op.py:30-40
    assert K == K2, f'Inner dim mismatch: {K} != {K2}'   # op.py:41
    out = x.new_empty((M, out_n))
    dev = _current_device()
    need = _workspace_bytes(dev, M, Nw, Kw, transpose_b)
    ws = _workspace(need, zeroed=True, tag='w4').data_ptr() if need else 0
    flags = (_lib.W4_TRANSPOSE_B if transpose_b else 0) | (_lib.W4_WEIGHTS_SETTLED if _settled(w) else 0)
    rc = lib.jgq_w4_matmul(x.data_ptr(), _DT[x.dtype], w.data_ptr(), zero.data_ptr(), scale.data_ptr(),
                           _ZS[zero.dtype], out.data_ptr(), M, Nw, Kw, flags, ws, need, _raw_stream(dev))
    if rc:
        check(rc)
    return out if len(shape) == 2 else out.reshape(shape[:-1] + (out_n,))


class _QuantizedMatmul(torch.autograd.Function):
    """forward: x @ W ; backward w.r.t. x: y_bar @ W^T via the transposed kernel (op.py:71-81)."""

    @staticmethod
    def forward(ctx, x, w, zero, scale, transpose_b):
        ctx.save_for_backward(w, zero, scale)
        ctx.transpose_b = transpose_b
        return _launch(x, w, zero, scale, transpose_b)

    @staticmethod
    def backward(ctx, y_bar):
        w, zero, scale = ctx.saved_tensors
        return _launch(y_bar, w, zero, scale, not ctx.transpose_b), None, None, None, None


def _on_device(t):
    """A contiguous CUDA tensor for `t`; what already is one comes back as it is."""
    if type(t) is torch.Tensor and t.is_cuda:
        return t if t.is_contiguous() else t.contiguous()
    return _to_dev(t).contiguous()


def _needs_function(x, zero, scale):
    """Whether anything besides the values depends on the product: gradients, forward-mode tangents, a functorch
    transform, a trace or a tensor subclass.  Those go through the autograd function; a plain product is launched
    directly (12 us of host time per call instead of 20)."""
    return (type(x) is not torch.Tensor or type(zero) is not torch.Tensor or type(scale) is not torch.Tensor
            or forward_ad._current_level >= 0 or _functorch_active() is not None or _tracing() is not None
            or (torch.is_grad_enabled() and (x.requires_grad or zero.requires_grad or scale.requires_grad)))


def quantized_matmul(x, quantized_matrix, transpose_b=False):
    """x @ dequant(quantized_matrix) (or its transpose); result in x's dtype."""
    as_np = _is_np(x)
    xd = x if type(x) is torch.Tensor and x.is_cuda else _to_dev(x)
    if xd.dtype not in _DT:
        xd = xd.to(torch.float32)
    if getattr(quantized_matrix, 'bits', 4) == 3:
        # 3-bit storage: expanded once to the nibble layout the kernels read and kept with the matrix
        cached = getattr(quantized_matrix, '_int4', None)
        if cached is None:
            from .gptq import to_int4_layout
            cached = to_int4_layout(quantized_matrix)
            quantized_matrix._int4 = cached
        quantized_matrix = cached
    w = _on_device(quantized_matrix.int_weight)
    if w.dim() != 2 or quantized_matrix.contraction_axis != 0:
        raise ValueError('quantized_matmul expects a 2-D QuantizedMatrix packed along axis 0')
    zero, scale = quantized_matrix.zero, quantized_matrix.scale
    if type(zero) is not torch.Tensor or type(scale) is not torch.Tensor or zero.dtype not in _ZS or zero.dtype != scale.dtype:
        zero, scale = _to_dev(zero), _to_dev(scale)
        if zero.dtype not in _ZS or zero.dtype != scale.dtype:
            zero, scale = zero.to(torch.float32), scale.to(torch.float32)
    zero, scale = _on_device(zero), _on_device(scale)
    if _needs_function(xd, zero, scale):
        out = _QuantizedMatmul.apply(xd, w, zero, scale, bool(transpose_b))
    else:
        out = _launch(xd, w, zero, scale, bool(transpose_b))
    return _out(out, as_np)
